// fp64_ops_check.cu -- the scalar operations of rbm_pp_b200/csrc/fp64_ops.cuh on arrays, for tests/test_gpu_fp64_ops.py.
#include "fp64_ops.cuh"

__global__ void ops_kernel(int n, const double* a, const double* b, double* out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double y = recip(b[i]);
  out[i] = y;
  out[n + i] = quotient(a[i], b[i], y);
  out[3 * n + i] = sqrt_recip(fabs(b[i]), out[2 * n + i]);
}

// words y whose fraction is not the quotient (all 2^32 over the grid)
__global__ void fraction_kernel(unsigned long long* bad) {
  unsigned long long c = 0;
  for (unsigned long long y = blockIdx.x * blockDim.x + threadIdx.x; y < (1ull << 32); y += gridDim.x * blockDim.x)
    c += word_fraction((uint32_t)y) != __ddiv_rn((double)(uint32_t)y, 4294967295.0);
  if (c) atomicAdd(bad, c);
}

// a, b: n doubles; out: 4 n doubles; bad: one word (host memory).  Returns the CUDA error code.
extern "C" int fp64_ops_check(int n, const double* a, const double* b, double* out, unsigned long long* bad) {
  double* d = nullptr;
  cudaError_t e = cudaMalloc(&d, sizeof(double) * 6 * (size_t)n + sizeof(*bad));
  if (e) return e;
  unsigned long long* db = (unsigned long long*)(d + 6 * (size_t)n);
  e = cudaMemcpy(d, a, sizeof(double) * n, cudaMemcpyHostToDevice);
  if (!e) e = cudaMemcpy(d + n, b, sizeof(double) * n, cudaMemcpyHostToDevice);
  if (!e) e = cudaMemset(db, 0, sizeof(*bad));
  if (!e) {
    ops_kernel<<<(n + 255) / 256, 256>>>(n, d, d + n, d + 2 * (size_t)n);
    fraction_kernel<<<1480, 256>>>(db);
    e = cudaGetLastError();
  }
  if (!e) e = cudaMemcpy(out, d + 2 * (size_t)n, sizeof(double) * 4 * n, cudaMemcpyDeviceToHost);
  if (!e) e = cudaMemcpy(bad, db, sizeof(*bad), cudaMemcpyDeviceToHost);
  cudaFree(d);
  return e;
}
