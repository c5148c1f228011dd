// bidiag.cuh -- what the kernels of the bidiagonal route share (bidiag.cu, bdapply.cu).
#pragma once
#include "tebd_internal.cuh"

namespace tebd {
namespace {

__device__ __forceinline__ bool on_route(int p) { return p == kPathBidiag || p == kPathBidiagT; }

// The matrix that is bidiagonalised, M x N with M >= N, in place in S.X (ld M):
// Theta itself (m x n) or, on the transposed route, Theta^H (n x m).
__device__ __forceinline__ void bd_dims(const Compact &cp, int p, int &M, int &N) {
  M = p == kPathBidiagT ? cp.n : cp.m;
  N = p == kPathBidiagT ? cp.m : cp.n;
}

// Where Theta's copy lies in S.aux, behind k_gebrd's workspace (units of 16 bytes): the
// right reflectors, the fixed-point matrix, the panel's vectors, the current column and row,
// the posted norms.
__host__ __device__ __forceinline__ size_t bd_theta_at(int M, int N) {
  const size_t Mp = (M + 31) / 32 * 32, Np = (N + 31) / 32 * 32;
  return (size_t)N * N + Mp * Np + 17 * (Mp + Np) + 128;
}

// bdws layout of one bond (doubles): d (n), e (n), sigma (kk), then from an even
// offset the inverse-iteration scratch U0, U1, U2, PV, Y (2n x K each), the
// eigenvectors Z (2n x K) and the left vectors Yu (m x K complex, 16-byte aligned)
__host__ __device__ __forceinline__ size_t bd_scratch(int n, int kk) {
  return ((size_t)2 * n + kk + 1) & ~(size_t)1;
}

// Whether a value of the K kept ones lies within 64 ulps of the next, by a whole warp (values
// below 64 ulps of the largest are left out: their vectors weigh as little).
__device__ __forceinline__ bool bd_clustered(const double *sig, int K) {
  const double near = 64.0 * 2.220446049250313e-16 * sig[0];
  bool close = false;
  for (int i = threadIdx.x & 31; i + 1 < K; i += 32) close |= sig[i] > near && sig[i] - sig[i + 1] <= near;
  return __any_sync(0xffffffffu, close);
}

}  // namespace
}  // namespace tebd
