// The one-CTA L x L routines of the block Krylov solvers on matrices of the caller's (tests/test_gpu_small_algebra.py).
#include <cuda_runtime.h>

#include "small.cuh"

namespace bdda {
namespace {

template <typename R>
__global__ void __launch_bounds__(kSmallThreads) k_lu(const double2* a, double2* b, int L, int full, int* ok) {
  using M = typename SmallMat<R>::M;
  extern __shared__ __align__(16) unsigned char raw[];
  M* A = reinterpret_cast<M*>(raw);
  M* B = A + L * L;
  int* piv = reinterpret_cast<int*>(B + L * L);
  sm_load(A, a, L * L);
  sm_load(B, b, L * L);
  __syncthreads();
  const bool good = sm_lu_solve<R>(A, B, L, L, full != 0, piv + kMaxL, piv);
  sm_store(b, B, L * L);
  if (threadIdx.x == 0) *ok = good;
}

template <typename R>
__global__ void __launch_bounds__(kSmallThreads) k_chol(const double2* h, double2* r, double2* ri, int L, int* ok) {
  using M = typename SmallMat<R>::M;
  extern __shared__ __align__(16) unsigned char raw[];
  M *H = reinterpret_cast<M*>(raw), *Rm = H + L * L, *Ri = Rm + L * L;
  sm_load(H, h, L * L);
  __syncthreads();
  const bool good = sm_chol_inv<R>(Rm, Ri, H, L);
  __syncthreads();
  sm_store(r, Rm, L * L);
  sm_store(ri, Ri, L * L);
  if (threadIdx.x == 0) *ok = good;
}

// host matrices (column-major complex FP64) in, results in place; the CUDA error
template <class Run> int on_device(double* x, double* y, double* z, int L, int* ok, Run run) {
  const size_t n = sizeof(double2) * L * L;
  double2* d = nullptr;
  cudaError_t e = cudaMalloc(&d, 3 * n + sizeof(int));
  if (e != cudaSuccess) return (int)e;
  double* host[3] = {x, y, z};
  int* dok = reinterpret_cast<int*>(d + 3 * L * L);
  for (int i = 0; i < 3 && e == cudaSuccess; ++i)
    if (host[i]) e = cudaMemcpy(d + i * L * L, host[i], n, cudaMemcpyHostToDevice);
  if (e == cudaSuccess) {
    run(d, d + L * L, d + 2 * L * L, dok, 3 * (int)n + 2 * kMaxL * (int)sizeof(int));
    e = cudaDeviceSynchronize();
  }
  for (int i = 0; i < 3 && e == cudaSuccess; ++i)
    if (host[i]) e = cudaMemcpy(host[i], d + i * L * L, n, cudaMemcpyDeviceToHost);
  if (e == cudaSuccess) e = cudaMemcpy(ok, dok, sizeof(int), cudaMemcpyDeviceToHost);
  cudaFree(d);
  return (int)e;
}

}  // namespace
}  // namespace bdda

using namespace bdda;

extern "C" {

// A X = B; df: double-float arithmetic
int lu(double* a, double* b, int L, int full, int df, int* ok) {
  return on_device(a, b, nullptr, L, ok, [&](double2* da, double2* db, double2*, int* dok, int smem) {
    auto* k = df ? k_lu<dfl> : k_lu<double>;
    cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    k<<<1, kSmallThreads, smem>>>(da, db, L, full, dok);
  });
}

// H = R^H R and R^-1
int chol(double* h, double* r, double* ri, int L, int df, int* ok) {
  return on_device(h, r, ri, L, ok, [&](double2* dh, double2* dr, double2* dri, int* dok, int smem) {
    auto* k = df ? k_chol<dfl> : k_chol<double>;
    cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    k<<<1, kSmallThreads, smem>>>(dh, dr, dri, L, dok);
  });
}

}  // extern "C"
