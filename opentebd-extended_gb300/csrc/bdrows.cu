// bdrows.cu -- step 5 of the bidiagonal route (bidiag.cu): small rows of the singular
// vectors to their own size.
//
// The fixed-point steps leave U and V accurate to about 1e-16 of the largest entry, the
// same in every row.  FormGamma1 and FormGamma2 (local_operations_module.f90:381-430) divide
// the rows by Lambda0 and Lambda2, so that a row of 1e-8 would come out to 1e-8 of its size
// (a floating-point bidiagonalisation of such a graded Theta keeps 1e-15 to 1e-13).  Theta
// itself has its rows and columns to rounding of their own size, and its product with a
// vector keeps that:
//   1. entry (r, i) of U becomes (Theta V)(r, i) / sigma_i where the row's norm is at most
//      sigma_i and an eighth of the largest value (larger rows have nothing to gain); then
//      V from Theta^H U in the same way.
//   2. The vectors of small values are known up to rotations among them of eps sigma_0 /
//      sigma_i, which step 1 mixes into single rows (1e-12 for values of 1e-8).  Each set
//      is made orthonormal again: with G = U^H U, U <- U (I - T), T the part of G - I above
//      the diagonal and half of it, vectors of larger values first; the square of G - I is
//      below eps.  G(k, i), k < i, is off by eps sigma_0 / sigma_k at most, and only if step 1
//      changed column k: T's rows k from 2^-8 sigma_0 down to the smallest row of Theta
//      are formed.  A row stays as accurate as it was: its larger entries lie at smaller
//      sigma_i, later in the order.
// Below 2^-26 of the largest value, where that square would not be small, a row is replaced
// only if the change is below eps: norm sigma_0 <= sigma_i^2.  The values keep the bisection's
// accuracy, eps of the largest.
//
// The products are those of fixed.cuh, with Theta's rows (columns) scaled to one
// exponent each: 64 x 32 tiles, 4 x 2 outputs per thread, whose 96 integer multiply-adds
// per k hide 10 shared-memory wavefronts, so that the integer pipe bounds it.  Tiles without
// a row small enough for their values return at once.  Measured: rows of Gamma1 Lambda1
// against extended precision, Lambdas down to 1e-8 (1e-4), 320 x 320: 1e-8 -> 3e-15 (2e-12 ->
// 3e-15); 80 x 80: 8e-9 -> 6e-13 (1e-12 -> 3e-15).  32 bonds of 640 x 640, 128 vectors: 3.1 ms
// beside 65; 10 of 270 x 270, 90 vectors: 0.7 beside 8.2.
#include <algorithm>

#include "bidiag.cuh"
#include "fixed.cuh"

namespace tebd {

namespace {

// of one row (left) or column (right) of Theta: its norm and an exponent above it
struct Line {
  double norm;
  int e, pad;
};
__device__ __forceinline__ const double2 *theta_of(const Slot &S, size_t base) { return S.aux + base; }
__device__ __forceinline__ Line *lines_of(const Slot &S, size_t base, int M, int N, bool left) {
  return reinterpret_cast<Line *>(S.aux + base + (size_t)M * N) + (left ? 0 : M);
}

constexpr int kLines = 32;  // rows or columns per CTA

__global__ void __launch_bounds__(256) k_bd_lines(Slot *slots, const int *path) {
  const int s = blockIdx.y;
  const int route = path[s];
  if (!on_route(route)) return;
  const Slot S = slots[s];
  int M, N;
  bd_dims(*S.cp, route, M, N);
  const bool left = blockIdx.z == 0;
  const int l0 = blockIdx.x * kLines, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, lim = left ? M : N;
  if (l0 >= lim) return;  // uniform
  const size_t base = bd_theta_at(M, N);
  const double2 *T = theta_of(S, base);
  Line *out = lines_of(S, base, M, N, left);
  // in units of a power of two near the largest value, so that no square overflows
  const int sc = max(-1000, min(1000, ((__double2hiint(S.bdws[2 * N]) >> 20) & 0x7ff) - 1023));
  const double down = pow2(-sc), up = pow2(sc);
  __shared__ double part[8][kLines];
  __shared__ int top[8][kLines];
  auto put = [&](int l, double sum, int big) {  // 2^(big + 1) bounds the entries' parts, the root of their number more the norm
    const int parts = 2 * (left ? N : M);
    out[l] = Line{sqrt(sum) * up, big + 1 + (33 - __clz(parts)) / 2, 0};
  };
  auto field = [](double x) { return ((__double2hiint(x) >> 20) & 0x7ff) - 1023; };
  if (left) {  // lanes over the rows, warps over the columns
    double acc = 0.0;
    int big = -1023;
    for (int c = warp; c < N && l0 + lane < M; c += 8) {
      const double2 t = T[l0 + lane + (size_t)M * c];
      const double x = t.x * down, y = t.y * down;
      acc = fma(x, x, fma(y, y, acc));
      big = max(big, max(field(t.x), field(t.y)));
    }
    part[warp][lane] = acc;
    top[warp][lane] = big;
    __syncthreads();
    if (warp == 0 && l0 + lane < M) {
      for (int w = 1; w < 8; ++w) {
        acc += part[w][lane];
        big = max(big, top[w][lane]);
      }
      put(l0 + lane, acc, big);
    }
  } else {
    for (int c = l0 + warp; c < min(N, l0 + kLines); c += 8) {
      double acc = 0.0;
      int big = -1023;
      for (int r = lane; r < M; r += 32) {
        const double2 t = T[r + (size_t)M * c];
        const double x = t.x * down, y = t.y * down;
        acc = fma(x, x, fma(y, y, acc));
        big = max(big, max(field(t.x), field(t.y)));
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
      big = __reduce_max_sync(0xffffffffu, big);
      if (lane == 0) put(c, acc, big);
    }
  }
}

constexpr int kTR = 64, kTC = 32, kTK = 16;  // tile rows, vectors, inner step
constexpr int kFold = 256;  // most products per sum of cross terms: 2^59 each, with room

__device__ __forceinline__ bool replaced(double norm, double si, double s0) {
  return norm <= 0.125 * s0 && norm <= si && (si >= 1.4901161193847656e-08 * s0 || norm <= si * (si / s0));
}

// One problem's arrays: U (M x K) and V (N x K) of the matrix that was bidiagonalised, its
// values, and T of both sets (K x K each, in the inverse iteration's scratch)
struct Vectors {
  int M, N, K;
  double2 *u, *v, *t;
  const double *sig;
  __device__ __forceinline__ bool load(const Slot &S, int route, int kk, int cap) {
    if (!on_route(route)) return false;
    bd_dims(*S.cp, route, M, N);
    K = cap ? min(min(kk, N), S.cp->k) : min(kk, N);
    sig = S.bdws + 2 * N;
    double *base = S.bdws + bd_scratch(N, kk);
    u = reinterpret_cast<double2 *>(base + 12 * (size_t)N * K);
    v = route == kPathBidiagT ? reinterpret_cast<double2 *>(base + 10 * (size_t)N * K) : S.V;
    t = reinterpret_cast<double2 *>(base);
    return true;
  }
  // rows [ka, kb) of T, by the whole CTA: values below 2^-8 of the largest, down to the smallest
  // norm of a line (side 1: row, 0: column) that is not zero
  __device__ __forceinline__ void tail(const Slot &S, int side, int &ka, int &kb) const {
    __shared__ int first[2];
    __shared__ unsigned long long least;
    if (threadIdx.x < 2) first[threadIdx.x] = K;
    if (threadIdx.x == 0) least = ~0ull;
    __syncthreads();
    const Line *lines = lines_of(S, bd_theta_at(M, N), M, N, side);
    unsigned long long low = ~0ull;
    for (int l = threadIdx.x; l < (side ? M : N); l += blockDim.x) {
      const double v = lines[l].norm;
      if (v > 0.0) low = min(low, (unsigned long long)__double_as_longlong(v));
    }
    atomicMin(&least, low);
    __syncthreads();
    const double a = 0.00390625 * sig[0], b = __longlong_as_double((long long)least);
    for (int i = threadIdx.x; i < K; i += blockDim.x) {
      if (sig[i] < a) atomicMin(&first[0], i);
      if (!(sig[i] >= b)) atomicMin(&first[1], i);
    }
    __syncthreads();
    ka = first[0];
    kb = first[1];
  }
};

using Tile = Acc[4][2];  // rows tid % 16 + 16 q, vectors tid / 16 + 16 p

// acc = the tile of rows r0.. and vectors i0.. of A B, A(r, k) = a[r ar + k ak] (conjugated),
// in units of 2^(ex[r] - 62), B(k, i) = b[k + len i] in units of 2^-62
__device__ __forceinline__ void product(Tile &acc, const double2 *a, size_t ar, size_t ak, bool conj, const int *ex,
                                        const double2 *b, int lim, int K, int len, int r0, int i0) {
  __shared__ int4 As[kTK][kTR + 1], Bs[kTK][kTC + 1];
  const int tid = threadIdx.x, rg = tid & 15, cg = tid >> 4;
  for (int k0 = 0; k0 < len; k0 += kTK) {
    for (int e = tid; e < kTR * kTK; e += 256) {  // the index that is contiguous in memory runs fastest
      const int r = ar == 1 ? e % kTR : e / kTK, k = ar == 1 ? e / kTR : e % kTK;
      int4 v = make_int4(0, 0, 0, 0);
      if (r0 + r < lim && k0 + k < len) {
        double2 t = a[(r0 + r) * ar + (k0 + k) * ak];
        if (conj) t.y = -t.y;
        v = enc2(to_fix(t.x, 62 - ex[r]), to_fix(t.y, 62 - ex[r]));
      }
      As[k][r] = v;
    }
    for (int e = tid; e < kTC * kTK; e += 256) {
      const int k = e % kTK, c = e / kTK;
      int4 v = make_int4(0, 0, 0, 0);
      if (i0 + c < K && k0 + k < len) {
        const double2 x = b[k0 + k + (size_t)len * (i0 + c)];
        v = vec_entry(to_fix(x.x, 62), to_fix(x.y, 62));
      }
      Bs[k][c] = v;
    }
    __syncthreads();
#pragma unroll 2
    for (int k = 0; k < kTK; ++k) {
      int4 x[4], y[2];
#pragma unroll
      for (int q = 0; q < 4; ++q) x[q] = As[k][rg + 16 * q];
#pragma unroll
      for (int p = 0; p < 2; ++p) y[p] = Bs[k][cg + 16 * p];
#pragma unroll
      for (int p = 0; p < 2; ++p) {
        const int nh = -y[p].z, nl = -y[p].w;
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[q][p].add(x[q], y[p], nh, nl);
      }
    }
    if ((k0 + kTK) % kFold == 0) {
#pragma unroll
      for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int p = 0; p < 2; ++p) {  // the cross terms' upper part moves over, exactly
          Acc &s = acc[q][p];
          s.hr += s.xr >> 28;
          s.hi += s.xi >> 28;
          s.xr &= (1 << 28) - 1;
          s.xi &= (1 << 28) - 1;
        }
    }
    __syncthreads();
  }
}

// 1. the entries to be replaced of the left (right) vectors, in place
__global__ void __launch_bounds__(256, 2) k_bd_rows(Slot *slots, const int *path, int kk, int cap, int left) {
  const int s = blockIdx.z;
  const Slot S = slots[s];
  Vectors w;
  if (!w.load(S, path[s], kk, cap)) return;
  const int lim = left ? w.M : w.N, r0 = blockIdx.x * kTR, i0 = blockIdx.y * kTC, tid = threadIdx.x;
  if (r0 >= lim || i0 >= w.K) return;  // uniform
  const size_t at = bd_theta_at(w.M, w.N);
  const double2 *T = theta_of(S, at);
  const Line *lines = lines_of(S, at, w.M, w.N, left);
  {  // anything to do?  (the values descend)
    bool any = false;
    if (tid < kTR && r0 + tid < lim) any = replaced(lines[r0 + tid].norm, w.sig[i0], w.sig[0]);
    if (!__syncthreads_or(any)) return;
  }
  __shared__ int ex[kTR];
  if (tid < kTR) ex[tid] = r0 + tid < lim ? lines[r0 + tid].e : 0;
  __syncthreads();
  Tile acc;
  product(acc, T, left ? 1 : w.M, left ? w.M : 1, !left, ex, left ? w.v : w.u, lim, w.K, left ? w.N : w.M, r0, i0);
  double2 *out = left ? w.u : w.v;
#pragma unroll
  for (int p = 0; p < 2; ++p) {
    const int i = i0 + (tid >> 4) + 16 * p;
    if (i >= w.K) continue;
    const double si = w.sig[i];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int r = r0 + (tid & 15) + 16 * q;
      if (r >= lim || !(si > 0.0 && replaced(lines[r].norm, si, w.sig[0]))) continue;
      const longlong2 z = acc[q][p].value<1>();  // units of 2^(e - 61)
      const int e = ex[(tid & 15) + 16 * q] - 61;
      out[r + (size_t)lim * i] = make_double2(scalbn((double)z.x, e) / si, scalbn((double)z.y, e) / si);
    }
  }
}

// 2. T of both sets (side 0: V, 1: U)
__global__ void __launch_bounds__(256, 2) k_bd_gram(Slot *slots, const int *path, int kk, int cap) {
  const int s = blockIdx.z, side = blockIdx.x & 1;
  Vectors w;
  if (!w.load(slots[s], path[s], kk, cap)) return;
  const int r0 = (blockIdx.x >> 1) * kTR, i0 = blockIdx.y * kTC, tid = threadIdx.x;
  if (r0 >= w.K || i0 >= w.K || r0 >= i0 + kTC) return;  // uniform
  int ka, kb;
  w.tail(slots[s], side, ka, kb);
  if (r0 >= kb || r0 + kTR <= ka) return;  // uniform
  const double2 *x = side ? w.u : w.v;
  const int len = side ? w.M : w.N;
  __shared__ int ex[kTR];
  if (tid < kTR) ex[tid] = 0;
  __syncthreads();
  Tile acc;
  product(acc, x, len, 1, true, ex, x, w.K, w.K, len, r0, i0);
  double2 *T = w.t + (size_t)side * w.K * w.K;
  const double unit = pow2(-61);
#pragma unroll
  for (int p = 0; p < 2; ++p)
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int r = r0 + (tid & 15) + 16 * q, i = i0 + (tid >> 4) + 16 * p;
      if (r > i || i >= w.K || r < ka || r >= kb) continue;
      const longlong2 z = acc[q][p].value<1>();
      double2 t = make_double2((double)z.x * unit, (double)z.y * unit);
      if (r == i) t = make_double2(z.x ? 0.5 * (double)(z.x - (1ll << 61)) * unit : 0.0, 0.0);  // a zero vector stays
      T[r + (size_t)w.K * i] = t;
    }
}

// U <- U - U T in place: a CTA owns 32 rows and takes the vectors from the last on, as a
// vector needs only those before it and itself.  T is below 2^-26, so that FP32 products do.
constexpr int kFR = 32, kFC = 32;
__global__ void __launch_bounds__(256) k_bd_orthonormal(Slot *slots, const int *path, int kk, int cap) {
  const int s = blockIdx.y, side = blockIdx.z;
  Vectors w;
  if (!w.load(slots[s], path[s], kk, cap)) return;
  const int lim = side ? w.M : w.N, r0 = blockIdx.x * kFR, tid = threadIdx.x;
  if (r0 >= lim) return;  // uniform
  int ka, kb;
  w.tail(slots[s], side, ka, kb);
  double2 *x = side ? w.u : w.v;
  const double2 *T = w.t + (size_t)side * w.K * w.K;
  __shared__ float2 Us[kFC][kFR + 1], Ts[kFC][kFC + 1];
  const int r = tid & 31, c = tid >> 5;  // row; vectors c + 8 q
  for (int i0 = ka < kb ? (w.K - 1) / kFC * kFC : -1; i0 >= ka / kFC * kFC; i0 -= kFC) {
    float re[4] = {0.f, 0.f, 0.f, 0.f}, im[4] = {0.f, 0.f, 0.f, 0.f};
    for (int k0 = ka / kFC * kFC; k0 <= i0 && k0 < kb; k0 += kFC) {
      for (int q = c; q < kFC; q += 8) {
        double2 a = make_double2(0.0, 0.0), t = a;
        if (r0 + r < lim && k0 + q < w.K) a = x[r0 + r + (size_t)lim * (k0 + q)];
        if (k0 + r >= ka && k0 + r < kb && k0 + r <= i0 + q && i0 + q < w.K) t = T[k0 + r + (size_t)w.K * (i0 + q)];
        Us[q][r] = make_float2((float)a.x, (float)a.y);
        Ts[q][r] = make_float2((float)t.x, (float)t.y);
      }
      __syncthreads();
#pragma unroll 8
      for (int k = 0; k < kFC; ++k) {
        const float2 a = Us[k][r];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const float2 t = Ts[c + 8 * q][k];
          re[q] = fmaf(a.x, t.x, fmaf(-a.y, t.y, re[q]));
          im[q] = fmaf(a.x, t.y, fmaf(a.y, t.x, im[q]));
        }
      }
      __syncthreads();
    }
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (r0 + r < lim && i0 + c + 8 * q < w.K) {
        double2 &v = x[r0 + r + (size_t)lim * (i0 + c + 8 * q)];
        v = make_double2(v.x - (double)re[q], v.y - (double)im[q]);
      }
    __syncthreads();
  }
}

}  // namespace

// Theta's copy from k_gebrd and the records of its lines
size_t bd_rows_aux_elems(int M, int N) { return (size_t)M * N + M + N; }

int launch_bd_rows(tebd_handle *h, const BidiagBatch &b) {
  k_bd_lines<<<dim3((b.nmax + kLines - 1) / kLines, b.nb, 2), 256, 0, h->stream>>>(b.slots_d, b.path_d);
  TEBD_LAUNCHED(h);
  for (int left = 1; left >= 0; --left) {  // the left vectors from the right ones, then the right ones from these
    k_bd_rows<<<dim3((b.nmax + kTR - 1) / kTR, (b.kk + kTC - 1) / kTC, b.nb), 256, 0, h->stream>>>(
        b.slots_d, b.path_d, b.kk, b.cap, left);
    TEBD_LAUNCHED(h);
  }
  k_bd_gram<<<dim3(2 * ((b.kk + kTR - 1) / kTR), (b.kk + kTC - 1) / kTC, b.nb), 256, 0, h->stream>>>(
      b.slots_d, b.path_d, b.kk, b.cap);
  TEBD_LAUNCHED(h);
  k_bd_orthonormal<<<dim3((b.nmax + kFR - 1) / kFR, b.nb, 2), 256, 0, h->stream>>>(b.slots_d, b.path_d, b.kk, b.cap);
  TEBD_LAUNCHED(h);
  return check_cuda(h, cudaGetLastError(), "row accuracy launch");
}

}  // namespace tebd
