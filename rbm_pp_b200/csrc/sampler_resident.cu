// sampler_resident.cu -- kernels and launchers of the resident sampler (sampler_resident.cuh).
#include "sampler_resident.cuh"

namespace {

template <int NP, int PPW, int THREADS, int MINB>
__global__ void __launch_bounds__(THREADS, MINB)
    sampler_resident_kernel(const __grid_constant__ DevDims d, const __grid_constant__ DevTables t,
                            const __grid_constant__ DevParams p, const __grid_constant__ DevWalkers W,
                            const __grid_constant__ ROff o, int first) {
  resident_body<NP, PPW>(d, t, p, W, o, (int)blockIdx.x, first);
}

// Warps of one walker's block.  Few projections: control, theta and G warps per projection, in eight warps (two
// blocks of 128 registers a thread fit an SM) up to 12x12 and sixteen at 14x14, whose blocks fill an SM alone.  Many:
// control and enough consumers that none holds more than kResMaxPpw projections.
int resident_warps(const DevDims& d) {
  if (d.n_qp <= kResFew) {
    return 2 + d.n_qp * resident_shares(d.n_qp, d.Np, d.Np > 72 ? 16 : 8);
  }
  const int rounds = (d.n_qp + 14) / 15;
  return 1 + (d.n_qp + rounds - 1) / rounds;
}

}  // namespace

// Threads per block of the resident sampler for a context, 0 when it does not apply: real units, the block sizes of
// the even lattices up to 14x14, and every inverse block of a walker in one SM's shared memory.
int rbmpp_resident_threads(const DevDims& d, int max_smem) {
  if (d.skew || d.alphac) return 0;
  switch (d.Np) {
    case 8: case 18: case 32: break;
    case 50: case 72: case 98:
      if (d.n_qp > kResFew) return 0;
      break;
    default: return 0;
  }
  if (d.n_qp > 15 * kResMaxPpw) return 0;
  const int w = resident_warps(d);
  // 512 bytes for the kernel's static shared memory
  return (long long)resident_layout(d.N, d.n_mp, d.alphar, w).total + 512 <= max_smem ? 32 * w : 0;
}

// Threads of a batched launch's blocks that suit every context of it, and their shared memory (the larger block
// size for N/2 = 98 or when the smaller one leaves a warp more than kResMaxPpw projections).
int rbmpp_resident_batch_threads(const DevDims& d) {
  return d.Np > 72 || d.n_qp > 7 * kResMaxPpw ? 512 : 256;
}
size_t rbmpp_resident_smem(const DevDims& d, int threads) {
  return resident_layout(d.N, d.n_mp, d.alphar, threads / 32).total;
}

cudaError_t rbmpp_launch_sampler_resident(const DevDims& d, const DevTables& t, const DevParams& p, const DevWalkers& W,
                                          int first, int threads, cudaStream_t st) {
  const ROff o = resident_layout(d.N, d.n_mp, d.alphar, threads / 32);
  const size_t smem = o.total;
#define LAUNCH(NP, PPW, TH, MB)                                                                          \
  do {                                                                                                   \
    cudaError_t e = cudaFuncSetAttribute(sampler_resident_kernel<NP, PPW, TH, MB>,                       \
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);        \
    if (e != cudaSuccess) return e;                                                                      \
    rbmpp_note_launch();                                                                                 \
    sampler_resident_kernel<NP, PPW, TH, MB><<<d.nw, threads, smem, st>>>(d, t, p, W, o, first);         \
    return cudaGetLastError();                                                                           \
  } while (0)
  if (d.n_qp <= kResFew) switch (d.Np) {
      case 8: LAUNCH(8, 1, 256, 2);
      case 18: LAUNCH(18, 1, 256, 2);
      case 32: LAUNCH(32, 1, 256, 2);
      case 50: LAUNCH(50, 1, 256, 2);
      case 72: LAUNCH(72, 1, 256, 2);
      case 98: LAUNCH(98, 1, 512, 1);
    }
  else switch (d.Np) {
      case 8: LAUNCH(8, kResMaxPpw, 512, 1);
      case 18: LAUNCH(18, kResMaxPpw, 512, 1);
      case 32: LAUNCH(32, kResMaxPpw, 512, 1);
    }
#undef LAUNCH
  return cudaErrorInvalidValue;
}
