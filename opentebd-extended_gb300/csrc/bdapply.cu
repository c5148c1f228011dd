// bdapply.cu -- step 4 of the bidiagonal route (bidiag.cu): the singular vectors of B
// back-transformed by the reflectors, U = Q [Ub; 0] and V = P Vb, the ZUNMBR part of
// ZGESVD (local_operations_module.f90:322-345).
//
// Each kept column y is independent: y <- H(0) ... H(n-1) y, H(j) = I - tau_j v_j v_j^H,
// the last reflector first.  In FP64 (a warp per column, its y in memory) the kernel was
// bound by the FP64 pipe: 8 of its instructions per element and reflector, 136 cycles a
// warp.  Here the reflectors come in fixed point from gebrd.cu and y is held in fixed
// point (units of 2^-62, |y| <= 1) in shared memory, a product being three integer
// multiply-adds (fixed.cuh).  Four reflectors at a time, as I - V T V^H (T upper
// triangular, from k_bd_wy): y is read and written once per four, and the latency of
// the sums over the lanes is paid once.  A CTA holds kCols columns (as many as fit),
// each by kWarps / kCols warps, which walk the reflectors nearly together, so that each
// is read from L2 about once per CTA.  Rounding: 2^-62 per block and element.
//
// Measured (GB300): 128 vectors a side of 32 matrices of 640 x 640, 38.3 -> 13.8 ms; 90 of
// 10 of 270 x 270, 2.55 -> 0.71 ms; 256 of 12 of 1024 x 1024 (double-float before), 29.8 ->
// 26.3 ms.  Bound by the integer pipe with a partly empty last wave; beyond 800 rows
// shared memory holds 8 columns and the warps of a column wait for one another.
#include <algorithm>

#include "bidiag.cuh"
#include "fixed.cuh"

namespace tebd {

namespace {

constexpr int kWarps = 16;
constexpr size_t kSmem = 200 * 1024;

// y in shared memory: x + 8 + 2^31 as one 64-bit integer, whose high word and (low word
// - 2^31) >> 4 are the halves that a product takes
constexpr long long kOff = 8 + 0x80000000ll;
struct Y {
  long long re, im;
};
__device__ __forceinline__ int4 as_entry(const Y &y) {  // as a vector entry
  return make_int4((int)(y.re >> 32), (int)((unsigned)y.re ^ 0x80000000u) >> 4, (int)(y.im >> 32),
                   (int)((unsigned)y.im ^ 0x80000000u) >> 4);
}

constexpr int kB = 4;      // reflectors per block
constexpr int kWy = 11;    // entries of a block's record: T by columns (10), then its exponent
__device__ __forceinline__ int t_at(int a, int b) { return b * (b + 1) / 2 + a; }  // a <= b

// records of the left side's blocks, then the right side's, behind U in S.aux (the
// bidiagonalisation's fixed-point matrix is free by now)
__device__ __forceinline__ int4 *wy_at(const Slot &S, int n, bool left) {
  return reinterpret_cast<int4 *>(S.aux) + (size_t)n * n + (left ? 0 : (size_t)kWy * ((n + kB - 1) / kB));
}

// T of each block of reflectors, one warp per block: the products v_a^H v_b as integer
// sums over the lanes, then LAPACK's ZLARFT recurrence T(0:b, b) = -tau_b T (V^H v_b).
__global__ void __launch_bounds__(128) k_bd_wy(Slot *slots, const int *path, int sides) {
  const int s = blockIdx.y;
  const int route = path[s];
  if (!on_route(route)) return;
  const Slot S = slots[s];
  int m, n;
  bd_dims(*S.cp, route, m, n);
  const bool left = blockIdx.z == 1;
  const int blk = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  const int nref = left ? n : n - 1, len = left ? m : n, j0 = kB * blk;
  if (j0 >= nref) return;
  const int cnt = min(kB, nref - j0);
  const int4 *R = left ? reinterpret_cast<const int4 *>(S.X) : reinterpret_cast<const int4 *>(S.aux);
  const double2 *taus = left ? S.tau : S.taup;
  Acc g[6];  // (0,1) (0,2) (1,2) (0,3) (1,3) (2,3)
  for (int r = (left ? j0 : j0 + 1) + lane; r < len; r += 32) {
    int4 v[kB];
#pragma unroll
    for (int a = 0; a < kB; ++a) v[a] = R[(size_t)len * (j0 + min(a, cnt - 1)) + r];
    int q = 0;
#pragma unroll
    for (int b = 1; b < kB; ++b) {
      const int4 e = make_int4(v[b].y, v[b].x >> 4, v[b].w, v[b].z >> 4);
#pragma unroll
      for (int a = 0; a < b; ++a) g[q++].add_conj(v[a], e, -e.x, -e.y);
    }
  }
  double2 G[6];
  const double unit = pow2(-61);
#pragma unroll
  for (int q = 0; q < 6; ++q) {
    longlong2 w = g[q].value<1>();
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      w.x += __shfl_xor_sync(0xffffffffu, w.x, o);
      w.y += __shfl_xor_sync(0xffffffffu, w.y, o);
    }
    G[q] = make_double2((double)w.x * unit, (double)w.y * unit);
  }
  double2 T[kB * (kB + 1) / 2];
  double big = 0.0;
#pragma unroll
  for (int b = 0; b < kB; ++b) {
    const double2 tau = b < cnt ? taus[j0 + b] : make_double2(0.0, 0.0);
    T[t_at(b, b)] = tau;
#pragma unroll
    for (int a = 0; a < b; ++a) {
      double2 acc = make_double2(0.0, 0.0);
#pragma unroll
      for (int c = a; c < b; ++c) acc = cadd(acc, cmul(T[t_at(a, c)], G[b * (b - 1) / 2 + c]));
      acc = cmul(tau, acc);
      T[t_at(a, b)] = make_double2(-acc.x, -acc.y);
    }
  }
#pragma unroll
  for (int q = 0; q < kB * (kB + 1) / 2; ++q) big = fmax(big, fmax(fabs(T[q].x), fabs(T[q].y)));
  const int e = max(0, (__double2hiint(big) >> 20) - 1022);  // |T| < 2^e; tau is 0 or at least 1 in size
  int4 *out = wy_at(S, n, left) + (size_t)kWy * blk;
  if (lane < kB * (kB + 1) / 2) {
    double2 t = make_double2(0.0, 0.0);
#pragma unroll
    for (int q = 0; q < kB * (kB + 1) / 2; ++q)
      if (q == lane) t = T[q];
    out[lane] = enc2(to_fix(t.x, 61 - e), to_fix(t.y, 61 - e));
  } else if (lane == 10) {
    out[10] = make_int4(e, 0, 0, 0);
  }
}

template <int kCols>
__global__ void __launch_bounds__(kWarps * 32, 1) k_bd_apply(Slot *slots, const int *path, int kk, int cap, int sides) {
  constexpr int kPer = kWarps / kCols;  // warps per column
  const int s = blockIdx.y;
  const int route = path[s];
  if (!on_route(route)) return;
  const Slot S = slots[s];
  int m, n;
  bd_dims(*S.cp, route, m, n);
  const int K = cap ? min(min(kk, n), S.cp->k) : min(kk, n);
  const int groups = gridDim.x / sides;
  const bool left = sides == 2 && (int)blockIdx.x >= groups;  // right vectors first
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int mine = warp / kPer, sub = warp % kPer, i = (blockIdx.x - (left ? groups : 0)) * kCols + mine;
  if (i - mine >= K) return;  // uniform per CTA
  const bool live = i < K;
  const int len = left ? m : n;
  extern __shared__ Y ys[];
  __shared__ long long part[kCols][kPer][2 * kB];
  __shared__ longlong2 fs[kWarps][kB];
  Y *y = ys + (size_t)len * mine;
  double *base = S.bdws + bd_scratch(n, kk);
  const int2 *Z = reinterpret_cast<const int2 *>(base) + ((size_t)(left ? K : 0) + i) * n;  // from k_bd_orth
  const int t0 = lane + 32 * sub, step = 32 * kPer;
  if (live)
    for (int r = t0; r < len; r += step) {
      long long z = 0;
      if (r < n) z = dec(Z[r].x, Z[r].y);
      y[r] = Y{z + kOff, kOff};
    }
  auto together = [&]() {  // the column's warps
    if (kPer > 1)
      asm volatile("bar.sync %0, %1;" ::"r"(1 + mine), "r"(32 * kPer) : "memory");
    else
      __syncwarp();
  };
  if (!live) return;  // a whole column's warps
  together();
  const int4 *R = left ? reinterpret_cast<const int4 *>(S.X) : reinterpret_cast<const int4 *>(S.aux);
  const int4 *wy = wy_at(S, n, left);
  const int nref = left ? n : n - 1;
  for (int blk = (nref + kB - 1) / kB - 1; blk >= 0; --blk) {
    const int j0 = kB * blk, r0 = left ? j0 : j0 + 1, cnt = min(kB, nref - j0);
    const int4 *v[kB];
#pragma unroll
    for (int a = 0; a < kB; ++a) v[a] = R + (size_t)len * (j0 + min(a, cnt - 1));
    const int4 *rec = wy + (size_t)kWy * blk;
    int4 t[kB];  // row a = lane & 3 of T
    const int a = lane & 3, eT = __ldcg(rec + 10).x;
#pragma unroll
    for (int b = 0; b < kB; ++b) t[b] = b >= a ? __ldcg(rec + t_at(a, b)) : make_int4(8, 0, 8, 0);
    Acc w[kB];
#pragma unroll 2
    for (int r = r0 + t0; r < len; r += step) {
      int4 x[kB];
#pragma unroll
      for (int b = 0; b < kB; ++b) x[b] = __ldg(v[b] + r);
      const int4 e = as_entry(y[r]);
      const int nh = -e.x, nl = -e.y;
#pragma unroll
      for (int b = 0; b < kB; ++b) w[b].add_conj(x[b], e, nh, nl);
    }
    long long q[2 * kB];  // V^H y in units of 2^-61
#pragma unroll
    for (int b = 0; b < kB; ++b) {
      const longlong2 z = w[b].value<1>();
      q[2 * b] = z.x;
      q[2 * b + 1] = z.y;
    }
#pragma unroll
    for (int h = 4; h >= 1; h >>= 1) {  // lane 4 c ends with the sum of value c
      const bool upper = lane & (4 * h);
#pragma unroll
      for (int c = 0; c < h; ++c) {
        const long long send = upper ? q[c] : q[c + h];
        q[c] = (upper ? q[c + h] : q[c]) + __shfl_xor_sync(0xffffffffu, send, 4 * h);
      }
    }
    q[0] += __shfl_xor_sync(0xffffffffu, q[0], 2);
    q[0] += __shfl_xor_sync(0xffffffffu, q[0], 1);
    if ((lane & 3) == 0) part[mine][sub][lane >> 2] = q[0];
    together();
    {  // f_a = sum_b T_ab w_b in units of 2^(eT - 59)
      Acc f;
#pragma unroll
      for (int b = 0; b < kB; ++b) {
        long long wr = 0, wi = 0;
#pragma unroll
        for (int c = 0; c < kPer; ++c) {
          wr += part[mine][c][2 * b];
          wi += part[mine][c][2 * b + 1];
        }
        const int4 e = vec_entry(wr, wi);
        f.add(t[b], e, -e.z, -e.w);
      }
      if (lane < kB) fs[warp][a] = f.value<1>();
    }
    together();
    // y -= V f, f scaled up to 61 bits
    long long big = 0;
    longlong2 f[kB];
#pragma unroll
    for (int b = 0; b < kB; ++b) {
      f[b] = fs[warp][b];
      big |= (f[b].x ^ (f[b].x >> 63)) | (f[b].y ^ (f[b].y >> 63));
    }
    const int z = min(max(__clzll(big) - 2, 0), max(0, 3 + eT));
    const int up = 5 + eT - z;  // units of f: 2^(eT - 59 - z); of y: 2^-62
    int4 fe[kB];
#pragma unroll
    for (int b = 0; b < kB; ++b) fe[b] = vec_entry(f[b].x << z, f[b].y << z);
    const long long half = 1ll << (27 - up);
#pragma unroll 2
    for (int r = r0 + t0; r < len; r += step) {
      int4 x[kB];
#pragma unroll
      for (int b = 0; b < kB; ++b) x[b] = __ldg(v[b] + r);
      Acc u;
#pragma unroll
      for (int b = 0; b < kB; ++b) u.add(x[b], fe[b], -fe[b].z, -fe[b].w);
      Y d = y[r];
      d.re -= (u.hr << up) + ((u.xr + half) >> (28 - up));
      d.im -= (u.hi << up) + ((u.xi + half) >> (28 - up));
      y[r] = d;
    }
    together();
  }
  // left -> Yu (scratch), right -> S.V (Theta route) or scratch (Theta^H route: z's, free by now)
  double2 *out = left ? reinterpret_cast<double2 *>(base + 6 * (size_t)(2 * n) * K) + (size_t)m * i
                      : (route == kPathBidiagT ? reinterpret_cast<double2 *>(base + 10 * (size_t)n * K) : S.V) + (size_t)n * i;
  const double unit = pow2(-62);
  for (int r = t0; r < len; r += step)
    out[r] = make_double2((double)(y[r].re - kOff) * unit, (double)(y[r].im - kOff) * unit);
}

}  // namespace

int launch_bd_apply(tebd_handle *h, const BidiagBatch &b) {
  // as many columns per CTA as shared memory holds, at most one per warp
  int cols = kWarps;
  while (cols > 1 && sizeof(Y) * (size_t)b.nmax * cols > kSmem) cols /= 2;
  const size_t smem = sizeof(Y) * (size_t)b.nmax * cols;
  const int sides = b.right_only ? 1 : 2;
  k_bd_wy<<<dim3((b.nmax + 4 * kB - 1) / (4 * kB), b.nb, sides), 128, 0, h->stream>>>(b.slots_d, b.path_d, sides);
  TEBD_LAUNCHED(h);
  auto go = [&](auto kern) {
    int rc = check_cuda(h, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem),
                        "back-transformation shared memory");
    if (rc) return rc;
    kern<<<dim3(sides * ((b.kk + cols - 1) / cols), b.nb), kWarps * 32, smem, h->stream>>>(b.slots_d, b.path_d, b.kk,
                                                                                          b.cap, sides);
    TEBD_LAUNCHED(h);
    return check_cuda(h, cudaGetLastError(), "back-transformation launch");
  };
  switch (cols) {
    case 16: return go(k_bd_apply<16>);
    case 8: return go(k_bd_apply<8>);
    case 4: return go(k_bd_apply<4>);
    case 2: return go(k_bd_apply<2>);
    default: return go(k_bd_apply<1>);
  }
}

}  // namespace tebd
