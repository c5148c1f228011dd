// bdorth.cu -- step 3b of the bidiagonal route (bidiag.cu): the singular vectors that
// inverse iteration gave, re-orthogonalised in order of descending sigma, which
// restores orthogonality inside clusters of close values (what DSTEIN does after
// DBDSQR's part of ZGESVD, local_operations_module.f90:322-345).
//
// The right vectors (even entries of z) and the left ones (odd entries) are two sets of
// real vectors.  One at a time, each against all before it, a vector cost three cluster
// barriers and FP64 sums (an FP64 instruction takes its SM 17 cycles): 28 us a vector.
// Here eight at a time, in 64-bit fixed point (fixed.cuh; units of 2^-62): the panel's
// dot products with all earlier vectors, one exchange between the CTAs, the
// subtraction, then the panel itself by the Cholesky factor of its Gram matrix; all
// of it again while a vector lost more than half of its squared norm in either part
// (the "twice is enough" test of Daniel, Gragg, Kaufman and Stewart).  A cluster of CTAs
// splits the rows of one set.
//
// Measured: 128 vectors of 32 bonds, n = 640: 6.8 -> 0.91 ms; 256 of 32, n = 1024, in the
// double-float form: 17.4 -> 2.3; 90 of 10, n = 270: 2.6 -> 0.32.
#include <cooperative_groups.h>
#include <math.h>

#include <algorithm>

#include "bidiag.cuh"
#include "fixed.cuh"

namespace tebd {

namespace {

constexpr int kThreads = 512, kWarps = kThreads / 32;
constexpr int kPan = 8;  // vectors per panel
constexpr int kMaxC = 8;
constexpr int kRounds = 6;  // most rounds of a panel
// smallest pivot of the Gram matrix: far above its rounding (2^-60), so that a vector that
// kept only 1e-7 or less of its norm comes out 1e7 times larger and is resolved by the
// next round
constexpr double kPivot = 1e-14;

// an entry of the panel in shared memory: x + 8 + 2^31 (see bdapply.cu)
constexpr long long kOff = 8 + 0x80000000ll;
__device__ __forceinline__ int p_hi(long long z) { return (int)(z >> 32); }
__device__ __forceinline__ int p_lo(long long z) { return (int)((unsigned)z ^ 0x80000000u) >> 4; }

// real sums as fixed.cuh's: h of high x high, x of the cross terms
struct RAcc {
  long long h = 0, x = 0;
  __device__ __forceinline__ void add(int ah, int al, int bh, int bl) {
    mw(h, ah, bh);
    mw(x, ah, bl);
    mw(x, al, bh);
  }
  template <int kUp>
  __device__ __forceinline__ long long value() const {
    constexpr int dn = 28 - kUp;
    return (long long)((unsigned long long)h << kUp) + ((x + (1ll << (dn - 1))) >> dn);
  }
};

__host__ __device__ __forceinline__ int rows_of(int n, int C) { return ((n + C - 1) / C + 31) / 32 * 32; }
__host__ __device__ __forceinline__ int splits(int rows) {  // parts of the earlier vectors per row group
  const int g = rows / 32;
  return g >= kWarps ? 1 : kWarps / g;
}
// shared memory: the panel (rows x 8), the coefficients (K x 8 pairs of ints), the
// subtraction's partial sums
__host__ __device__ __forceinline__ size_t orth_smem(int n, int K, int C) {
  const size_t rows = rows_of(n, C);
  // splits(r) r is at most max(r, 512), but not monotone in r: the batch's smaller problems
  // may need more than its largest
  return sizeof(long long) * kPan * (rows + (size_t)K + (rows > 32 * kWarps ? rows : 32 * kWarps));
}
constexpr int kMostK = 2048;  // coefficients of more vectors stay in global memory

}  // namespace

// z's sets in fixed point, column by column: element (j, i) of set p at
// Zi[(p K + i) n + j], the layout the kernel below and the back-transformation read
__global__ void __launch_bounds__(256) k_bd_zfix(Slot *slots, const int *path, int kk, int cap, int second) {
  __shared__ double tile[2][32][33];
  const int s = blockIdx.z;
  const int route = path[s];
  if (!on_route(route)) return;
  const Slot S = slots[s];
  int m, n;
  bd_dims(*S.cp, route, m, n);
  const int K = cap ? min(min(kk, n), S.cp->k) : min(kk, n);
  const int i0 = blockIdx.x * 32, j0 = blockIdx.y * 32;
  if (i0 >= K || j0 >= n || (second && !bd_clustered(S.bdws + 2 * n, K))) return;  // uniform
  double *base = S.bdws + bd_scratch(n, kk);
  const double *Z = base + 5 * (size_t)(2 * n) * K;
  int2 *Zi = reinterpret_cast<int2 *>(base);
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  for (int y = ty; y < 64; y += 8) {
    const int j = j0 + (y >> 1), i = i0 + tx;
    if (j < n && i < K) tile[y & 1][y >> 1][tx] = Z[(size_t)(2 * j + (y & 1)) * K + i];
  }
  __syncthreads();
  for (int y = ty; y < 64; y += 8) {
    const int p = y >> 5, i = i0 + (y & 31), j = j0 + tx;
    if (j < n && i < K) Zi[((size_t)p * K + i) * n + j] = enc(to_fix(tile[p][tx][y & 31], 62));
  }
}

__global__ void __launch_bounds__(kThreads, 1) k_bd_orth(Slot *slots, const int *path, int kk, int cap, int d_in_smem,
                                                        int second) {
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  const int C = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
  const int s = blockIdx.y, part = blockIdx.x / C;  // part 0: v = z[2j], 1: u = z[2j+1]
  const int route = path[s];
  if (!on_route(route)) return;  // uniform per cluster
  const Slot S = slots[s];
  int m, n;
  bd_dims(*S.cp, route, m, n);
  const int K = cap ? min(min(kk, n), S.cp->k) : min(kk, n);
  if (second && !bd_clustered(S.bdws + 2 * n, K)) return;  // uniform per cluster
  double *base = S.bdws + bd_scratch(n, kk);
  int2 *Zi = reinterpret_cast<int2 *>(base) + (size_t)part * K * n;
  // the CTAs' dot products, two buffers in turn: [buffer][CTA][vector][panel vector]
  double *own_ws = base + 12 * (size_t)n * K + 2 * (size_t)m * K;
  long long *xch = reinterpret_cast<long long *>(own_ws) + (size_t)part * 2 * C * (K + kPan) * kPan;
  const int rows = rows_of(n, C), j0 = rank * rows, nr = max(0, min(n - j0, rows));
  extern __shared__ long long sm[];
  long long *P = sm;                                      // [8][rows]
  long long *sub = P + kPan * rows;                       // [split][8][rows]
  int2 *D = d_in_smem ? reinterpret_cast<int2 *>(sub + (size_t)splits(rows) * kPan * rows)  // [K][8]
                      : reinterpret_cast<int2 *>(own_ws + 4 * (size_t)kMaxC * (K + kPan) * kPan + (size_t)part * kPan * K);
  __shared__ double G[kPan][kPan], Ri[kPan][kPan], lost[kPan];
  __shared__ int again;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int nsplit = splits(rows);
  int turn = 0;
  auto slot_of = [&](int r, int c) { return xch + (((size_t)(turn & 1) * C + r) * (K + kPan) + c) * kPan; };
  auto exchange = [&]() {
    if (C > 1)
      cluster.sync();
    else
      __syncthreads();
  };
  for (int i = 0; i < K; i += kPan) {
    const int np = min(kPan, K - i);
    for (int e = tid; e < kPan * rows; e += kThreads) {
      const int q = e / rows, r = e - q * rows;
      long long x = 0;
      if (q < np && r < nr) {
        const int2 z = Zi[(size_t)(i + q) * n + j0 + r];
        x = dec(z.x, z.y);
      }
      P[e] = x + kOff;
    }
    __syncthreads();
    for (int round = 0; round < kRounds; ++round) {
      bool more = false;
      // ---- against all earlier vectors ----
      if (i > 0) {
        for (int c = 2 * warp; c < i; c += 2 * kWarps) {  // two earlier vectors (i is even)
          RAcc acc[2][kPan];
          const int2 *z0 = Zi + (size_t)c * n + j0, *z1 = z0 + n;
#pragma unroll 2
          for (int r = lane; r < nr; r += 32) {
            const int2 a = z0[r], b = z1[r];
            const int al = a.x >> 4, bl = b.x >> 4;
#pragma unroll
            for (int q = 0; q < kPan; ++q) {
              const long long p = P[q * rows + r];
              const int ph = p_hi(p), pl = p_lo(p);
              acc[0][q].add(a.y, al, ph, pl);
              acc[1][q].add(b.y, bl, ph, pl);
            }
          }
          long long t[2 * kPan];
#pragma unroll
          for (int q = 0; q < 2 * kPan; ++q) t[q] = acc[q / kPan][q % kPan].value<1>();
#pragma unroll
          for (int h = kPan; h >= 1; h >>= 1) {  // lanes 2 q, 2 q + 1 end with the sum of value q
            const bool upper = lane & (2 * h);
#pragma unroll
            for (int q = 0; q < h; ++q) {
              const long long send = upper ? t[q] : t[q + h];
              t[q] = (upper ? t[q + h] : t[q]) + __shfl_xor_sync(0xffffffffu, send, 2 * h);
            }
          }
          t[0] += __shfl_xor_sync(0xffffffffu, t[0], 1);
          const int q = lane >> 1;
          if (!(lane & 1)) slot_of(rank, c + q / kPan)[q % kPan] = t[0];
        }
        if (warp < kPan) {  // squared norms of the panel's vectors, behind the earlier vectors' slots
          RAcc acc;
          for (int r = lane; r < nr; r += 32) {
            const long long p = P[warp * rows + r];
            acc.add(p_hi(p), p_lo(p), p_hi(p), p_lo(p));
          }
          long long t = acc.value<1>();
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
          if (lane == 0) slot_of(rank, i)[warp] = t;
        }
        exchange();
        for (int e = tid; e < kPan * i; e += kThreads) {
          long long t = 0;
          for (int r = 0; r < C; ++r) t += __ldcg(slot_of(r, 0) + e);
          const int2 z = enc(t);  // units of 2^-61
          D[e] = make_int2(z.y, z.x >> 4);
        }
        if (tid == 0) again = 0;
        __syncthreads();
        if (warp < np) {  // did the projection take more than half of a squared norm?
          float acc = 0.f;
          for (int c = lane; c < i; c += 32) {
            const float d = (float)D[c * kPan + warp].x * (1.0f / 536870912.0f);  // high halves: units of 2^-29
            acc += d * d;
          }
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
          long long t = 0;
          for (int r = 0; r < C; ++r) t += __ldcg(slot_of(r, i) + warp);
          if (lane == 0 && acc > 0.5f * (float)t * 4.3368087e-19f) again = 1;  // t in units of 2^-61
        }
        const int groups = rows / 32;
        for (int task = warp; task < groups * nsplit; task += kWarps) {
          const int g = task % groups, h = task / groups, r = 32 * g + lane;
          const int c0 = (int)((long long)i * h / nsplit), c1 = (int)((long long)i * (h + 1) / nsplit);
          RAcc acc[kPan];
          if (r < nr) {
            const int2 *z = Zi + j0 + r;
#pragma unroll 4
            for (int c = c0; c < c1; ++c) {
              const int2 a = z[(size_t)c * n];
              const int al = a.x >> 4;
              const int4 *d = reinterpret_cast<const int4 *>(D + c * kPan);
#pragma unroll
              for (int q = 0; q < kPan / 2; ++q) {
                const int4 e = d[q];
                acc[2 * q].add(a.y, al, e.x, e.y);
                acc[2 * q + 1].add(a.y, al, e.z, e.w);
              }
            }
          }
#pragma unroll
          for (int q = 0; q < kPan; ++q) sub[((size_t)h * kPan + q) * rows + r] = acc[q].value<3>();
        }
        __syncthreads();
        for (int e = tid; e < kPan * rows; e += kThreads) {
          long long t = 0;
          for (int h = 0; h < nsplit; ++h) t += sub[(size_t)h * kPan * rows + e];
          P[e] -= t;
        }
        ++turn;
        more = again;
        __syncthreads();
      }
      // ---- the panel itself: P <- P R^-1, R the Cholesky factor of its Gram matrix ----
      for (int e = warp; e < kPan * (kPan + 1) / 2; e += kWarps) {
        int b = 0, a = e;
        while (a > b) a -= ++b;  // e = b (b + 1) / 2 + a, a <= b
        RAcc acc;
        for (int r = lane; r < nr; r += 32) {
          const long long x = P[a * rows + r], y = P[b * rows + r];
          acc.add(p_hi(x), p_lo(x), p_hi(y), p_lo(y));
        }
        long long t = acc.value<1>();
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        if (lane == 0) slot_of(rank, K + a)[b] = t;
      }
      exchange();
      if (tid < kPan * kPan) {
        const int a = min(tid / kPan, tid % kPan), b = max(tid / kPan, tid % kPan);
        long long t = 0;
        for (int r = 0; r < C; ++r) t += __ldcg(slot_of(r, K + a) + b);
        G[a][b] = G[b][a] = (double)t * pow2(-61);
      }
      __syncthreads();
      if (warp == 0) {
        // lane q < 8 holds column q of the factor; rows in order: R(k, q)
        const int q = lane & 7;
        double g[kPan], ri[kPan];
#pragma unroll
        for (int k = 0; k < kPan; ++k) g[k] = G[k][q];
        const double own = G[q][q];
        double left = own;  // what the earlier rows leave of the squared norm
        double rinv = 0.0;  // 1 / R(q, q)
#pragma unroll
        for (int k = 0; k < kPan; ++k) {
          // pivot of row k, from lane k; a smaller one than kPivot is raised to it (a
          // zero vector stays zero)
          double inv = 0.0;
          if (q == k && own > 0.0) inv = rsqrt(fmax(left, kPivot));
          if (q == k) rinv = inv;
          inv = __shfl_sync(0xffffffffu, inv, k);
          const double rk = g[k] * inv;  // R(k, q), q > k
          if (q > k) left = fma(-rk, rk, left);
          // trailing Gram entries: g(l, q) -= R(k, l) R(k, q)
#pragma unroll
          for (int l = 0; l < kPan; ++l) {
            const double rl = __shfl_sync(0xffffffffu, rk, l);
            if (l > k && q >= l) g[l] = fma(-rl, rk, g[l]);
          }
          g[k] = q > k ? rk : (q == k ? left * inv : 0.0);
        }
        // R^-1 by columns: lane q solves R x = e_q (g[k] = R(k, q) of every lane q)
#pragma unroll
        for (int k = 0; k < kPan; ++k) ri[k] = 0.0;
#pragma unroll
        for (int k = kPan - 1; k >= 0; --k) {
          double acc = k == q ? 1.0 : 0.0;
#pragma unroll
          for (int l = k + 1; l < kPan; ++l) {
            const double rkl = __shfl_sync(0xffffffffu, g[k], l);
            acc = fma(-rkl, ri[l], acc);
          }
          const double d = __shfl_sync(0xffffffffu, rinv, k);
          ri[k] = k <= q ? acc * d : 0.0;
        }
        if (lane < kPan) {
#pragma unroll
          for (int k = 0; k < kPan; ++k) Ri[k][q] = ri[k];
          lost[q] = own > 0.0 && left < fmax(0.5 * own, kPivot) ? 1.0 : 0.0;
        }
      }
      __syncthreads();
#pragma unroll
      for (int q = 0; q < kPan; ++q) more = more || lost[q] != 0.0;
      for (int r = tid; r < rows; r += kThreads) {
        double x[kPan];
#pragma unroll
        for (int q = 0; q < kPan; ++q) x[q] = (double)(P[q * rows + r] - kOff);
#pragma unroll
        for (int q = kPan - 1; q >= 0; --q) {
          double t = 0.0;
#pragma unroll
          for (int k = 0; k <= q; ++k) t = fma(x[k], Ri[k][q], t);
          P[q * rows + r] = to_fix(t, 0) + kOff;
        }
      }
      ++turn;
      __syncthreads();
      if (!more) break;
    }
    for (int e = tid; e < np * rows; e += kThreads) {
      const int q = e / rows, r = e - q * rows;
      if (r < nr) Zi[(size_t)(i + q) * n + j0 + r] = enc(P[e] - kOff);
    }
    __syncthreads();  // the CTA's own rows of the panel, before they are read as earlier vectors
  }
}

// its share of bdws, behind the left vectors: the exchange buffers of both sets, and
// coefficients that shared memory cannot hold
size_t bd_orth_ws_doubles(int K) { return 4 * (size_t)kMaxC * (K + kPan) * kPan + 2 * (size_t)kPan * K; }

// Both kernels on the batch; C CTAs per set, or the autotuner's number.  second: the second
// pass, only problems with clustered values; *clusters: C, 0 before the first pass.
int launch_bd_orth(tebd_handle *h, const BidiagBatch &b, int second, int *clusters) {
  const int sides = b.right_only ? 1 : 2;
  int nbd = 0;
  for (int s = 0; s < b.nb; ++s) nbd += b.path_h[s] != kPathQRJ;
  k_bd_zfix<<<dim3((b.kk + 31) / 32, (b.nmax + 31) / 32, b.nb), 256, 0, h->stream>>>(b.slots_d, b.path_d, b.kk, b.cap,
                                                                                               second);
  TEBD_LAUNCHED(h);
  constexpr size_t kSmemMax = 220 * 1024;
  int rc = check_cuda(h, cudaFuncSetAttribute(k_bd_orth, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemMax),
                      "orthogonalisation shared memory");
  if (rc) return rc;
  cudaLaunchConfig_t cfg = {};
  cfg.blockDim = dim3(kThreads, 1, 1);
  cfg.stream = h->stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  const int K = std::min(b.kk, b.nmax), d_in_smem = K <= kMostK;
  auto fits = [&](int c) {
    cfg.gridDim = dim3(sides * c, b.nb, 1);
    attr[0].val.clusterDim.x = c;
    cfg.dynamicSmemBytes = orth_smem(b.nmax, d_in_smem ? K : 0, c);
    int ncl = 0;
    if (cfg.dynamicSmemBytes > kSmemMax ||
        cudaOccupancyMaxActiveClusters(&ncl, (const void *)k_bd_orth, &cfg) != cudaSuccess) {
      cudaGetLastError();
      ncl = 0;
    }
    return ncl;
  };
  // Enough CTAs to fill the GPU once, at least 64 rows each; more where shared memory
  // asks for it.
  int C = *clusters;
  for (int c = 1; c <= kMaxC && !*clusters; c *= 2)
    if (fits(c) >= 1 && (C == 0 || (nbd * sides * c <= 152 && b.nmax >= 64 * c))) C = c;
  const TuneParams tp = tune_lookup(h, b.dfp ? 1 : 0, b.nmax, b.nb);
  if (tp.orth_cluster > 0 && !*clusters) {
    if (tp.orth_cluster <= kMaxC && fits(tp.orth_cluster) >= 1)
      C = tp.orth_cluster;
    else
      tune_reject(h);
  }
  if (C == 0) return set_error(h, TEBD_ERR_CUDA, "orthogonalisation: no cluster size fits");
  *clusters = C;
  cfg.gridDim = dim3(sides * C, b.nb, 1);
  attr[0].val.clusterDim.x = C;
  cfg.dynamicSmemBytes = orth_smem(b.nmax, d_in_smem ? K : 0, C);
  rc = check_cuda(h, cudaLaunchKernelEx(&cfg, k_bd_orth, b.slots_d, b.path_d, b.kk, b.cap, d_in_smem, second), "orthogonalisation launch");
  TEBD_LAUNCHED(h);
  return rc;
}

}  // namespace tebd
