// The helpers of csrc/fp64_util.cuh, one value per thread, for test_gpu_fp64_util.py.
#include "fp64_util.cuh"

__global__ void probe_kernel(const double* a, const double* b, long long n, double* div, double* rec, double* root,
                             int* index) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    if (div) div[i] = fp64::div_markstein(a[i], b[i]);
    if (rec) rec[i] = fp64::recip_newton(b[i]);
    if (root) root[i] = fp64::sqrt_markstein(b[i]);
    if (index) index[i] = fp64::pade_index(fp64::finite_od(a[i]));
  }
}

// device pointers; null outputs are left out
extern "C" int probe(const double* a, const double* b, long long n, double* div, double* rec, double* root,
                     int* index) {
  probe_kernel<<<1024, 256>>>(a, b, n, div, rec, root, index);
  const cudaError_t e = cudaGetLastError();
  return (int)(e != cudaSuccess ? e : cudaDeviceSynchronize());
}
