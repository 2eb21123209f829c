// sampler_resident_batch.cu -- the resident sampler (sampler_resident.cuh) over the walkers of several contexts.
#include "sampler_resident.cuh"

namespace {

// Walkers of several contexts in one launch: block b runs walker sched[b].y of context sched[b].x.
template <int THREADS, int MINB>
__global__ void __launch_bounds__(THREADS, MINB)
    resident_batch_kernel(const BatchInst* __restrict__ inst, const int2* __restrict__ sched, int first,
                          long long* __restrict__ cycles) {
  __shared__ BatchInst bi;
  __shared__ ROff o;
  const int2 job = sched[blockIdx.x];
  if (threadIdx.x == 0) {
    bi = inst[job.x];
    o = resident_layout(bi.d.N, bi.d.n_mp, bi.d.alphar, THREADS / 32);
  }
  __syncthreads();
  const long long c0 = clock64();
  const bool few = bi.d.n_qp <= kResFew;
#define RES(NP, PPW) resident_body<NP, PPW>(bi.d, bi.t, bi.p, bi.W, o, job.y, first)
  switch (bi.d.Np) {
    case 8:
      if (few) RES(8, 1);
      else RES(8, kResMaxPpw);
      break;
    case 18:
      if (few) RES(18, 1);
      else RES(18, kResMaxPpw);
      break;
    case 32:
      if (few) RES(32, 1);
      else RES(32, kResMaxPpw);
      break;
    case 50: RES(50, 1); break;
    case 72: RES(72, 1); break;
    case 98:
      if constexpr (THREADS == 512) RES(98, 1);
      break;
  }
#undef RES
  if (cycles && threadIdx.x == 0) cycles[blockIdx.x] = clock64() - c0;
}

}  // namespace

cudaError_t rbmpp_launch_resident_batch(const BatchInst* inst, const int2* sched, int n_blocks, int first, int threads,
                                        size_t smem, long long* cycles, cudaStream_t st) {
#define LAUNCH(TH, MB)                                                                                          \
  do {                                                                                                          \
    cudaError_t e = cudaFuncSetAttribute(resident_batch_kernel<TH, MB>, cudaFuncAttributeMaxDynamicSharedMemorySize, \
                                         (int)smem);                                                            \
    if (e != cudaSuccess) return e;                                                                             \
    rbmpp_note_launch();                                                                                        \
    resident_batch_kernel<TH, MB><<<n_blocks, TH, smem, st>>>(inst, sched, first, cycles);                      \
    return cudaGetLastError();                                                                                  \
  } while (0)
  if (threads == 256) LAUNCH(256, 2);
  if (threads == 512) LAUNCH(512, 1);
#undef LAUNCH
  return cudaErrorInvalidValue;
}

// Resident blocks per SM of the batched launch (0 if it cannot launch).
int rbmpp_resident_batch_occupancy(int threads, size_t smem) {
  int nb = 0;
  const void* f = threads == 256 ? (const void*)resident_batch_kernel<256, 2> : (const void*)resident_batch_kernel<512, 1>;
  if (cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return 0;
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, f, threads, smem) == cudaSuccess ? nb : 0;
}
