// gebrd.cu -- Householder bidiagonalisation of a compacted Theta (or charge block,
// or Gram) on the tensor cores: step 1 of the bidiagonal route (bidiag.cu), in place
// of the ZGEBRD part of ZGESVD (local_operations_module.f90:322-345).
//
// Why integers: the chip has 1.06 TFLOP/s of FP64 (an FP64 instruction occupies its SM
// for 17 cycles), and the two matrix-vector products per column that a
// bidiagonalisation cannot avoid are half of its flops.  In FP64 they bound the kernel
// at a tenth of the memory rate.  Here the trailing matrix is held as 64-bit
// fixed-point numbers (scaled by a power of two above its Frobenius norm: 2^-62 of it
// is the resolution, finer than FP64's own rounding of the norm-sized entries), as a
// pair of 32-bit halves, and a product is three 32 x 32 -> 64 bit multiply-adds (high x
// high, and the two cross terms with 28 bits of the low halves; 1.1 cycles each), the
// sums exact and bounded by the norms, rounded once per entry of the result.  Twelve
// of them per complex multiply-add take 14 cycles where four FP64 ones take 68.
// (Digit products on the tensor cores, mma.sync m16n8k16 with the digits of the vector
// as its 16 rows, measured slower: a matrix element used once does not pay for its
// split into digits.)  What is used many times, the panel's update of the trailing
// matrix, does run on the tensor cores: eight signed 8-bit digits per number as FP16
// integers, 45 of the 64 digit pairs, exact integer sums in the FP32 accumulators.
//
// The scheme is ZLABRD's: inside a panel of 8 columns the trailing matrix keeps its
// panel-start values A0 and the current one is A0 - V Y^H - X U^H; the panel end
// applies the update, 16 x 8 tiles with the digits of L = [V X] and R = [Y U] (16
// vectors: one MMA k step).  The corrections of the current row and column, of z and
// of w, and the dot products with the panel's vectors are integer sums too, so the
// FP64 pipe is left with the reflectors' scalars and about 30 operations per row and
// column.  One thread-block cluster per problem; CTA k owns the 8-row and 8-column
// blocks congruent to k.  It computes z = A0^H v for its columns and w = A0 u for its
// rows alone (and the 16 dot products, all of them, for itself), all of the raw vector,
// so the reflector's scale factor can follow later and a column needs two cluster
// barriers: the current column (then row) and its squared norm are posted before each.
// The reflectors are left in fixed point (units of 2^-62) for the back-transformation:
// v_i from its 1 on in column i of S.X, u_i in column i of the N x N array at S.aux.
//
// Measured (GB300, 2070 MHz), a batch of 32 matrices of 640 x 640: 148 ms with FP64
// dot products and FP64 tensor-core updates, 40 ms now; 10 of 270 x 270: 23.2 -> 5.5
// ms; 12 of 1024 x 1024 (double-float before): 157 -> 74 ms.  What bounds it: for
// hundreds of columns the integer pipe (a complex multiply-add of a warp takes 14
// cycles; 17 to 21 measured with its loads, 6.5 TB/s where the matrices exceed the L2),
// below that the latency of a column: two cluster barriers, four __syncthreads and the
// reflector's FP64 scalars, about 15 us.
#include <cooperative_groups.h>
#include <cuda_fp16.h>
#include <math.h>

#include <algorithm>

#include "bidiag.cuh"
#include "fixed.cuh"

namespace tebd {

namespace {

constexpr int kP = 8;         // columns per panel: V and X of a panel fill the 16 k of one MMA
constexpr int kMaxC = 8;      // CTAs per cluster
constexpr int kThreads = 512;
constexpr int kChunk = 256;   // most columns per sum of the row products: the cross terms stay in 64 bits
constexpr int kPairs = 8;     // pairs of 8-row blocks whose L fragments are staged at a time
constexpr unsigned long long kBias = 0x8080808080808080ull;  // signed digits as unsigned bytes

__host__ __device__ __forceinline__ int up(int x, int q) { return (x + q - 1) / q * q; }
// rows (columns) one CTA of C owns of n, in 8-blocks
__host__ __device__ __forceinline__ int own_count(int n, int C) { return up(up(n, 8) / 8, C) / C * 8; }

__device__ __forceinline__ double2 ldc(const double2 *p) { return __ldcg(p); }

__device__ __forceinline__ double wsum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// ZLARFG's scalars from alpha and ||x||^2: beta (real), tau, and 1/(alpha - beta).  One
// FP64 instruction holds a warp's scheduler for 64 cycles, so the root and the two
// reciprocals start from FP32 ones (rsqrtf, 1 / x) and take two Newton steps each.
__device__ __forceinline__ double newton_rsqrt(double x) {  // x > 0, exponent even-scaled into FP32's range
  const int e = ((__double2hiint(x) >> 20) - 1023) & ~1;
  const double m = __hiloint2double(__double2hiint(x) - (e << 20), __double2loint(x));  // [1, 4)
  double y = (double)rsqrtf((float)m);
  const double h = 0.5 * m;
  y = y * fma(-h * y, y, 1.5);
  y = y * fma(-h * y, y, 1.5);
  return __hiloint2double(__double2hiint(y) - ((e >> 1) << 20), __double2loint(y));
}
__device__ __forceinline__ double newton_rcp(double x) {  // x > 0
  const int e = (__double2hiint(x) >> 20) - 1023;
  const double m = __hiloint2double(__double2hiint(x) - (e << 20), __double2loint(x));  // [1, 2)
  double y = (double)(1.0f / (float)m);
  y = fma(y, fma(-m, y, 1.0), y);
  y = fma(y, fma(-m, y, 1.0), y);
  return __hiloint2double(__double2hiint(y) - (e << 20), __double2loint(y));
}
__device__ __forceinline__ void larfg(double2 alpha, double xn2, double &beta, double2 &tau, double2 &sc) {
  const double b2 = fma(alpha.x, alpha.x, fma(alpha.y, alpha.y, xn2));
  if (b2 < 1e-280) {  // nothing left (or squares out of range): H = I
    beta = alpha.x;
    tau = make_double2(0.0, 0.0);
    sc = make_double2(1.0, 0.0);
    return;
  }
  if (xn2 == 0.0 && alpha.y == 0.0) {
    beta = alpha.x;
    tau = make_double2(0.0, 0.0);
    sc = make_double2(1.0, 0.0);
    return;
  }
  const double r = newton_rsqrt(b2), ib = -copysign(r, alpha.x);
  beta = b2 * ib;
  tau = make_double2(fma(-alpha.x, ib, 1.0), -alpha.y * ib);
  const double dr = alpha.x - beta, iden = newton_rcp(fma(dr, dr, alpha.y * alpha.y));
  sc = make_double2(dr * iden, -alpha.y * iden);
}

__device__ __forceinline__ void mma(float (&d)[4], const uint4 a, unsigned b0, unsigned b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b0), "r"(b1));
}

// q - tau (q + scz z)
__device__ __forceinline__ double2 minus_reflected(longlong2 q, longlong2 z, double2 tau, double2 scz) {
  const double qr = (double)q.x, qi = (double)q.y, zr = (double)z.x, zi = (double)z.y;
  const double wr = fma(scz.x, zr, fma(-scz.y, zi, qr)), wi = fma(scz.x, zi, fma(scz.y, zr, qi));
  return make_double2(fma(-tau.x, wr, fma(tau.y, wi, qr)), fma(-tau.x, wi, fma(-tau.y, wr, qi)));
}

// two unsigned digit bytes (in bytes 2 s, 2 s + 1 of x) as a pair of FP16 digits:
// 0x6400 | b is 1024 + b, less 1152 the signed digit
__device__ __forceinline__ unsigned half_digits(unsigned x, int s) {
  const unsigned y = __byte_perm(x, 0x64646464u, s ? 0x4342 : 0x4140);
  __half2 h = *reinterpret_cast<const __half2 *>(&y);
  h = __hsub2(h, __halves2half2(__ushort_as_half(0x6480), __ushort_as_half(0x6480)));
  return *reinterpret_cast<unsigned *>(&h);
}

// digit bytes of two biased fixed-point numbers a, b: word q holds digits 2 q and
// 2 q + 1 of both
__device__ __forceinline__ void split_words(unsigned long long a, unsigned long long b, unsigned (&w)[4]) {
  const unsigned ah = (unsigned)(a >> 32), al = (unsigned)a, bh = (unsigned)(b >> 32), bl = (unsigned)b;
  w[0] = __byte_perm(ah, bh, 0x6273);
  w[1] = __byte_perm(ah, bh, 0x4051);
  w[2] = __byte_perm(al, bl, 0x6273);
  w[3] = __byte_perm(al, bl, 0x4051);
}
// their digits as FP16 pairs: d[p] holds digit p of both
__device__ __forceinline__ void split_pair(unsigned long long a, unsigned long long b, unsigned (&d)[8]) {
  unsigned w[4];
  split_words(a, b, w);
#pragma unroll
  for (int p = 0; p < 8; ++p) d[p] = half_digits(w[p >> 1], p & 1);
}

// Workspace of one problem, from S.aux (units of 16 bytes): U (N x N, read by the
// back-transformation), the fixed-point matrix (ld Mp, Np columns), the panel's [V X]
// (16 x ld Mp) and [Y U] (16 x ld Np), the raw current column and conjugated row, and
// the squared norms posted per warp of the cluster; with `keep` a copy of the matrix as it
// was behind them (bd_theta_at), for bdrows.cu.
static_assert(kThreads / 32 * kMaxC <= 128, "bd_theta_at");

// The problem, in shared memory: held in registers it would push the loops' own values
// into local memory.
struct Ctx {
  double2 *X, *tau, *taup;
  int4 *Pv;
  double *d, *e;
  int4 *A;             // fixed-point matrix
  // [V X], [Y U]: V, U in units of 2^-62, X, Y in units of 2^(eA - 61): with |tau| |v| <= 2
  // they are at most twice the matrix's norm, 2^62 units (coarser ones cost small singular
  // values: 512 x 512 of norm 6.5, values below 0.01 off by 2.5e-15 in units of 2^(eA - 58),
  // by 5e-16 now)
  int4 *Li, *Ri;
  double2 *col, *row;  // in units of 2^eA, so that their squares stay in range
  double *nl, *nr;
  int M, N, Mp, Np, C, rank, ownR, ownC, nnorm, eA;
  int lf_at, zc_at, zp_at, npb;  // shared memory, in 16-byte units
};
struct Scal {  // a reflector, written by one warp
  double2 tau, sc, scz;  // scz: sc in the units of the products' sums over A's
};

// shared memory, in 16-byte units: 16 panel coefficients (row i / column i+1), the 16
// dot products as coefficients, the dot products, the problem, the two reflectors, then
// the vector (one per entry), the panel update's L fragments (512 per pair of row
// blocks staged), and the products' sums per owned row or column: partial ones, four
// for the panel's correction of the row / column, four for that of z / w
extern __shared__ uint4 sh[];
constexpr int kRvec = 0, kSvec = 16, kDots = 32, kCtx = 48, kScal = 64, kVec = 72;
static_assert(sizeof(Ctx) <= 16 * (kScal - kCtx) && 2 * sizeof(Scal) <= 16 * (kVec - kScal), "shared memory layout");
__device__ __forceinline__ Ctx &ctx() { return *reinterpret_cast<Ctx *>(sh + kCtx); }
__device__ __forceinline__ Scal &scal(int k) { return reinterpret_cast<Scal *>(sh + kScal)[k]; }
__device__ __forceinline__ longlong2 *sums(int at) { return reinterpret_cast<longlong2 *>(sh + at); }
__device__ __forceinline__ const int4 *vector_at(int at) { return reinterpret_cast<const int4 *>(sh + at); }

__host__ __device__ __forceinline__ int pair_batch(int M, int C) {
  const int n = (own_count(M, C) / 8 + 1) / 2;
  return n < kPairs ? n : kPairs;
}
__host__ __device__ __forceinline__ int sum_slots(int M, int C) {
  return 32 * (2 * (kThreads / 32) + (own_count(M, C) + 31) / 32);
}
__host__ __device__ __forceinline__ size_t smem_bytes(int M, int C) {
  return 16 * ((size_t)kVec + up(M, 32) + 512 * pair_batch(M, C) + sum_slots(M, C) + 8 * (size_t)own_count(M, C));
}
constexpr size_t kSmemMax = 224 * 1024;

// a barrier for the vector and the coefficients: the last warp, busy with the
// reflector, only arrives
__device__ __forceinline__ void workers_sync() { asm volatile("bar.sync 1, %0;" ::"r"(kThreads) : "memory"); }
__device__ __forceinline__ void workers_arrive() { asm volatile("bar.arrive 1, %0;" ::"r"(kThreads) : "memory"); }
constexpr int kWarps = kThreads / 32, kWorkers = kWarps - 1;

// own index o -> global row / column of the CTA, and the smallest own index whose
// global index is >= x
__device__ __forceinline__ int glob(int o, int C, int rank) { return ((o >> 3) * C + rank) * 8 + (o & 7); }
__device__ __forceinline__ int first_own(int x, int C, int rank) {
  const int b = x >> 3;
  const int o = b <= rank ? 0 : (b - rank + C - 1) / C;
  return o * 8 + ((o * C + rank) == b ? (x & 7) : 0);
}

// D^H x for two columns of D (leading dimension ldd; entries [ka, kb), multiples of 32)
// by one warp, lanes over k, x in shared memory.  Lane 8 q returns value q: the real and
// imaginary part of column q / 2 in turn.
__device__ __forceinline__ long long columns_dot(const int4 *D, size_t ldd, int ka, int kb, int lane) {
  const int4 *vec = vector_at(kVec);
  Acc acc[2];
#pragma unroll 4
  for (int k = ka + lane; k < kb; k += 32) {
    const int4 a0 = __ldcg(D + k), a1 = __ldcg(D + ldd + k), v = vec[k];
    const int nh = -v.x, nl = -v.y;
    acc[0].add_conj(a0, v, nh, nl);
    acc[1].add_conj(a1, v, nh, nl);
  }
  const longlong2 x = acc[0].value<1>(), y = acc[1].value<1>();
  // sum over the lanes, halving the values that a lane is responsible for
  const bool u16 = lane & 16, u8 = lane & 8;
  long long t0 = u16 ? y.x : x.x, t1 = u16 ? y.y : x.y;
  t0 += __shfl_xor_sync(0xffffffffu, u16 ? x.x : y.x, 16);
  t1 += __shfl_xor_sync(0xffffffffu, u16 ? x.y : y.y, 16);
  long long t = u8 ? t1 : t0;
  t += __shfl_xor_sync(0xffffffffu, u8 ? t0 : t1, 8);
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  return t;
}

// sum over k in [ka, kb) of base[ldk k] vec[k], vec in shared memory
__device__ __forceinline__ void row_sum(Acc &acc, const int4 *base, size_t ldk, int ka, int kb, const int4 *vec) {
#pragma unroll 8
  for (int k = ka; k < kb; ++k) {
    const int4 v = vec[k];
    acc.add(__ldcg(base + ldk * k), v, -v.z, -v.w);
  }
}

// Phase A's products, a task per worker warp at a time: z = A0^H v for the CTA's own
// columns (two columns and one of `left_parts` parts of k per task) into the sums
// [part][column], the dot products of the panel's V, X with v, and quarters of the
// panel's correction of the current row, [Y U] rvec.  (The phases' functions are not
// inlined: each keeps its registers for its own loop.)
__device__ __forceinline__ int left_parts(int nk, int nz) {  // enough tasks for two rounds, at least 128 k each,
  const Ctx &x = ctx();                                       // as many as the sums have room for
  return max(1, min(min((2 * kWorkers + nz - 1) / max(1, nz), nk / 128), (x.zp_at - x.zc_at) / x.ownC));
}
__device__ __noinline__ void left_products(int i, bool panel, int warp, int lane) {
  const Ctx &x = ctx();
  const int C = x.C, rank = x.rank, Mp = x.Mp, Np = x.Np, ownC = x.ownC;
  const int ka = (i + 1) & ~31, o0 = first_own(i + 1, C, rank);
  const int first = o0 >> 1, nz = (ownC >> 1) - first, nd = panel ? 8 : 0, ob = o0 & ~7;
  const int np = panel ? 4 * ((ownC - ob + 31) / 32) : 0;
  const int parts = left_parts(Mp - ka, nz), len = up((Mp - ka + parts - 1) / parts, 32);
  longlong2 *zc = sums(x.zc_at), *zp = sums(x.zp_at);
  for (int task = warp; task < nz * parts + nd + np; task += kWorkers) {
    if (task < nz * parts + nd) {
      const bool dot = task >= nz * parts;
      const int part = dot ? 0 : task / nz, o = 2 * (dot ? task - nz * parts : first + task - part * nz);
      const int c = dot ? o : glob(o, C, rank);
      if (!dot && c >= Np) continue;
      const int k0 = ka + part * len, k1 = dot ? Mp : min(Mp, k0 + len);
      const long long out = columns_dot((dot ? x.Li : x.A) + (size_t)Mp * c, Mp, k0, k1, lane);
      if ((lane & 7) == 0)
        reinterpret_cast<long long *>((dot ? sums(kDots) : zc + part * ownC) + o)[lane >> 3] = out;
    } else {
      const int e = task - nd - nz * parts, o = ob + 32 * (e >> 2) + lane, c = glob(o, C, rank);
      if (o < ownC && c < Np) {
        Acc acc;
        row_sum(acc, x.Ri + c, Np, 4 * (e & 3), 4 * (e & 3) + 4, vector_at(kRvec));
        zp[(e & 3) * ownC + o] = acc.value<3>();
      }
    }
  }
}

// Phase B's: w = A0 u for the CTA's own rows, 32 rows x a chunk of columns per task, into
// [chunk][row]; the dot products of Y, U with u; quarters of [V X] rvec.
__device__ __forceinline__ int row_chunk_size(int nk, int groups) {  // two rounds of tasks
  const int want = (2 * kWorkers + groups - 1) / max(1, groups);
  return up(max(8, (nk + want - 1) / want), 8);
}
__device__ __noinline__ void right_products(int i, int warp, int lane) {
  const Ctx &x = ctx();
  const int C = x.C, rank = x.rank, Mp = x.Mp, Np = x.Np, ownR = x.ownR;
  const int ka = (i + 2) & ~31, ob = first_own(i + 1, C, rank) & ~7;
  const int groups = (ownR - ob + 31) / 32, nk = Np - ka;
  const int size = row_chunk_size(nk, groups), chunks = (nk + size - 1) / size;
  longlong2 *zc = sums(x.zc_at), *zp = sums(x.zp_at);
  for (int task = warp; task < groups * (chunks + 4) + 8; task += kWorkers) {
    if (task >= groups * chunks && task < groups * chunks + 8) {
      const int k = 2 * (task - groups * chunks);
      const long long out = columns_dot(x.Ri + (size_t)Np * k, Np, ka, Np, lane);
      if ((lane & 7) == 0) reinterpret_cast<long long *>(sums(kDots) + k)[lane >> 3] = out;
      continue;
    }
    const bool main = task < groups * chunks;
    const int e = main ? task : task - 8 - groups * chunks, ch = e / groups, gr = e - ch * groups;
    const int o = ob + 32 * gr + lane, r = glob(o, C, rank);
    if (o < ownR && r < Mp) {
      if (main) {
        longlong2 w = make_longlong2(0, 0);
        const int k1 = min(Np, ka + (ch + 1) * size);
        for (int k0 = ka + ch * size; k0 < k1; k0 += kChunk) {
          Acc acc;
          row_sum(acc, x.A + r, Mp, k0, min(k1, k0 + kChunk), vector_at(kVec));
          const longlong2 t = acc.value<1>();
          w.x += t.x;
          w.y += t.y;
        }
        zc[(ch * groups + gr) * 32 + lane] = w;
      } else {
        Acc acc;
        row_sum(acc, x.Li + r, Mp, 4 * ch, 4 * ch + 4, vector_at(kRvec));
        zp[ch * ownR + o] = acc.value<3>();
      }
    }
  }
}

// The panel's corrections of z (or w) by the dot products: quarter q of P svec, P (its
// leading dimension `lim`) the 16 vectors of the other side.  `own` owned rows of it.
__device__ __noinline__ void correct(bool left, int i, int warp, int lane) {
  const Ctx &x = ctx();
  const int C = x.C, rank = x.rank, own = left ? x.ownC : x.ownR, lim = left ? x.Np : x.Mp;
  const int4 *P = left ? x.Ri : x.Li;
  const int ob = first_own(i + 1, C, rank) & ~7, groups = (own - ob + 31) / 32;
  longlong2 *zq = sums(x.zp_at) + 4 * own;
  for (int task = warp; task < 4 * groups; task += kWarps) {
    const int o = ob + 32 * (task >> 2) + lane, q = task & 3, r = glob(o, C, rank);
    if (o < own && r < lim) {
      Acc acc;
      row_sum(acc, P + r, lim, 4 * q, 4 * q + 4, vector_at(kSvec));
      zq[q * own + o] = acc.value<3>();
    }
  }
}

// z - zq and q - zp of own index o: the sums of the panel's corrections taken off
__device__ __forceinline__ void take_off(longlong2 &z, longlong2 &q, int own, int o) {
  const longlong2 *zp = sums(ctx().zp_at) + o;
#pragma unroll
  for (int h = 0; h < 4; ++h) {
    q.x -= zp[h * own].x;
    q.y -= zp[h * own].y;
    z.x -= zp[(4 + h) * own].x;
    z.y -= zp[(4 + h) * own].y;
  }
}

// the biased digits of a stored fixed-point number
__device__ __forceinline__ unsigned long long digits_of(int lo, int hi) {
  return (unsigned long long)dec(lo, hi) + kBias;
}

// The panel's end: A0 -= L R^H for the CTA's own row blocks and the columns from q on, in
// fixed point.  16 x 8 tiles (a pair of own row blocks), the whole inner dimension in
// one MMA step.
__device__ __noinline__ void panel_update(int q, int warp, int lane) {
  const Ctx &cx = ctx();
  int4 *A = cx.A;
  const int4 *Li = cx.Li, *Ri = cx.Ri;
  const int Mp = cx.Mp, Np = cx.Np, C = cx.C, crank = cx.rank, npb = cx.npb, nwarp = kWarps;
  const int ob0 = first_own(q, C, crank) >> 3, ob1 = cx.ownR >> 3, cb0 = q >> 3, cb1 = up(cx.N, 8) >> 3;
  uint4 *Lf = sh + cx.lf_at;
          const int g = lane >> 2, t = lane & 3;
          const int npair = (ob1 - ob0 + 1) / 2;
          const int ncb = cb1 - cb0;
          auto row_a = [&](int pr) { return ((ob0 + 2 * pr) * C + crank) * 8 + g; };
          for (int pb = 0; pb < npair; pb += npb) {
            const int np = min(npb, npair - pb);
            __syncthreads();
            for (int f = warp; f < 2 * np; f += nwarp) {  // L fragments: even f real parts, odd f imaginary parts
              const int ra = row_a(pb + (f >> 1)), rb = ra + 8 * C;
              unsigned a0[8], a1[8], a2[8], a3[8];
              unsigned long long va[4], vb[4];
#pragma unroll
              for (int x = 0; x < 4; ++x) {
                const size_t k = (size_t)Mp * (4 * x + t);
                const int4 la = ra < Mp ? __ldcg(&Li[k + ra]) : make_int4(8, 0, 8, 0);
                const int4 lb = rb < Mp ? __ldcg(&Li[k + rb]) : make_int4(8, 0, 8, 0);
                va[x] = digits_of(f & 1 ? la.z : la.x, f & 1 ? la.w : la.y);
                vb[x] = digits_of(f & 1 ? lb.z : lb.x, f & 1 ? lb.w : lb.y);
              }
              split_pair(va[0], va[1], a0);
              split_pair(vb[0], vb[1], a1);
              split_pair(va[2], va[3], a2);
              split_pair(vb[2], vb[3], a3);
              uint4 *L = Lf + (size_t)(f >> 1) * 512 + (f & 1) * 32 + lane;
#pragma unroll
              for (int x = 0; x < 8; ++x) L[64 * x] = make_uint4(a0[x], a1[x], a2[x], a3[x]);
            }
            __syncthreads();
            // tasks: a column block and a share of the staged pairs
            const int split = min(np, max(1, nwarp / max(1, ncb)));
            for (int task = warp; task < ncb * split; task += nwarp) {
              const int cb = cb0 + task / split;
              unsigned br0[8], br1[8], bi0[8], bi1[8];
              {
                unsigned long long vr[4], vi[4];
#pragma unroll
              for (int x = 0; x < 4; ++x) {
                const int4 e = __ldcg(Ri + (size_t)(cb * 8 + g) + (size_t)Np * (4 * x + t));
                vr[x] = digits_of(e.x, e.y);
                vi[x] = digits_of(e.z, e.w);
              }
              split_pair(vr[0], vr[1], br0);
              split_pair(vr[2], vr[3], br1);
              split_pair(vi[0], vi[1], bi0);
              split_pair(vi[2], vi[3], bi1);
            }
              for (int pr = task % split; pr < np; pr += split) {
                const int ra = row_a(pb + pr), rb = ra + 8 * C;
                const uint4 *L = Lf + (size_t)pr * 512 + lane;
                int4 av[4];  // rows ra (x < 2) and rb, columns 2 t, 2 t + 1
#pragma unroll
                for (int x = 0; x < 4; ++x)
                  if ((x < 2 ? ra : rb) < Mp)
                    av[x] = __ldcg(&A[(x < 2 ? ra : rb) + (size_t)Mp * (cb * 8 + 2 * t + (x & 1))]);
                long long tr[4] = {0, 0, 0, 0}, ti[4] = {0, 0, 0, 0};
                int lr[4], li[4];
#pragma unroll
                for (int s = 0; s < 9; ++s) {
                  float dre[4] = {0.f, 0.f, 0.f, 0.f}, di1[4] = {0.f, 0.f, 0.f, 0.f}, di2[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                  for (int x = (s < 8 ? 0 : 1); x <= (s < 8 ? s : 7); ++x) {
                    const uint4 lre = L[64 * x], lim = L[64 * x + 32];
                    mma(dre, lre, br0[s - x], br1[s - x]);
                    mma(di1, lim, br0[s - x], br1[s - x]);
                    mma(di2, lre, bi0[s - x], bi1[s - x]);
                    mma(dre, lim, bi0[s - x], bi1[s - x]);
                  }
#pragma unroll
                  for (int x = 0; x < 4; ++x) {
                    const int re = (int)dre[x], im = (int)di1[x] - (int)di2[x];
                    if (s < 7) {
                      tr[x] = (tr[x] << 8) + re;
                      ti[x] = (ti[x] << 8) + im;
                    } else if (s == 7) {
                      lr[x] = re << 8;
                      li[x] = im << 8;
                    } else {
                      lr[x] += re;
                      li[x] += im;
                    }
                  }
                }
#pragma unroll
                for (int x = 0; x < 4; ++x)
                  if ((x < 2 ? ra : rb) < Mp) {
                    av[x] = enc2(dec(av[x].x, av[x].y) - (tr[x] << 3) - ((lr[x] + 4096) >> 13),
                               dec(av[x].z, av[x].w) - (ti[x] << 3) - ((li[x] + 4096) >> 13));
                  __stcg(&A[(x < 2 ? ra : rb) + (size_t)Mp * (cb * 8 + 2 * t + (x & 1))], av[x]);
                  }
              }
            }
          }
}

// an exponent e with the sum of the cnt posted squared norms < 2^(2 e), by the whole
// warp in integer instructions
__device__ __forceinline__ int norm_exponent(const double *n2, int cnt, int lane) {
  int hi[4] = {0, 0, 0, 0}, e = 0;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    if (lane + 32 * q < cnt) hi[q] = __double2hiint(__ldcg(n2 + lane + 32 * q));
    e = max(e, hi[q] >> 20);
  }
  e = __reduce_max_sync(0xffffffffu, e);
  unsigned m = 0;  // mantissas to 21 bits, rounded up
#pragma unroll
  for (int q = 0; q < 4; ++q)
    if (hi[q]) m += (((hi[q] & 0xfffff) | 0x100000) >> min(31, e - (hi[q] >> 20))) + 1;
  m = __reduce_add_sync(0xffffffffu, m);
  return (e - 1043 + 32 - __clz(m) + 1) >> 1;  // sum < m 2^(e - 1043)
}
static_assert(kThreads / 32 * kMaxC <= 128, "norm_exponent reads four values per lane");

// posts a warp's squared norm; `any` (uniform per warp): whether it has a part of it
__device__ __forceinline__ void post_norm(double *where, double acc, bool any, int warp, int lane) {
  if (any) acc = wsum(acc);
  if (lane == 0) where[ctx().rank * kWarps + warp] = any ? acc : 0.0;
}

// the reflector's scalars from alpha and the posted norms, by one warp; ez: exponent
// of the raw vector's unit
__device__ __noinline__ void reflector(int which, double2 alpha, int ez, int i, int lane) {
  const Ctx &x = ctx();
  const double *n2 = which ? x.nr : x.nl;
  double xn2 = 0.0;
  for (int q = lane; q < x.nnorm; q += 32) xn2 += __ldcg(n2 + q);
  xn2 = wsum(xn2);
  double beta;
  double2 tau, sc;
  larfg(alpha, xn2, beta, tau, sc);
  if (lane == 0) {
    const double zs = pow2(ez + 1);  // the sums' unit 2^(eA + ez - 61) over A's 2^(eA - 62)
    const double size = beta * pow2(x.eA);
    Scal &out = scal(which);
    out.tau = tau;
    out.sc = sc;
    out.scz = make_double2(sc.x * zs, sc.y * zs);
    if (x.rank == 0) {
      (which ? x.e : x.d)[i] = size;
      (which ? x.taup : x.tau)[i] = tau;
    }
  }
}

// conj of entry `at` of the panel's vector k as a coefficient (zero where unused)
__device__ __forceinline__ void coefficient(const int4 *P, size_t ld, int k, int at, bool use) {
  int4 v = make_int4(8, 0, 8, 0);
  if (use) v = __ldcg(P + ld * k + at);
  reinterpret_cast<int4 *>(sh + kRvec)[k] = vec_entry(dec(v.x, v.y), -dec(v.z, v.w));
}

// the raw vector's entries (lo, hi) of [ka, kp), zero elsewhere, by the worker warps
__device__ __forceinline__ void put_vector(const double2 *v, int ka, int kp, int lo, int hi, int ez, int tid) {
  int4 *vec = reinterpret_cast<int4 *>(sh + kVec);
  for (int r = ka + tid; r < kp; r += 32 * kWorkers) {
    long long xr = 0, xi = 0;
    if (r > lo && r < hi) {
      const double2 a = ldc(&v[r]);
      xr = to_fix(a.x, 62 - ez);
      xi = to_fix(a.y, 62 - ez);
    }
    vec[r] = vec_entry(xr, xi);
  }
}

// the 16 dot products as coefficients, those in use (by one warp)
__device__ __forceinline__ void dots_to_coefficients(bool use, int lane) {
  if (lane < 16) {
    const longlong2 d = use ? sums(kDots)[lane] : make_longlong2(0, 0);
    reinterpret_cast<int4 *>(sh + kSvec)[lane] = vec_entry(d.x, d.y);
  }
}

// y_i (panel column j) and row i of the current matrix, conjugated, for the own columns;
// ai: the first one's entry of A0.  Returns this thread's first entry of the row.
__device__ __noinline__ double2 finish_row(int i, int j, int4 ai, int tid) {
  const Ctx &x = ctx();
  const int C = x.C, rank = x.rank, ownC = x.ownC, N = x.N;
  const int oc = first_own(i + 1, C, rank);
  const int parts = left_parts(x.Mp - ((i + 1) & ~31), (ownC >> 1) - (oc >> 1));
  const double2 tau = scal(0).tau, scz = scal(0).scz;
  const double uA = pow2(-62);
  const longlong2 *zc = sums(x.zc_at);
  double acc = 0.0;
  double2 mine = make_double2(0.0, 0.0);
  for (int o = oc + tid; o < ownC; o += kThreads) {
    const int c = glob(o, C, rank);
    if (c >= N) continue;
    if (o != oc + tid) ai = __ldcg(&x.A[i + (size_t)x.Mp * c]);
    longlong2 q = make_longlong2(dec(ai.x, ai.y), -dec(ai.z, ai.w)), z = zc[o];  // q: conj of the row before H(i)
    for (int h = 1; h < parts; ++h) {
      z.x += zc[h * ownC + o].x;
      z.y += zc[h * ownC + o].y;
    }
    if (j > 0) take_off(z, q, ownC, o);
    // u = q - tau (q + scz z) in units of 2^(eA - 62); y = q - u
    const double2 u = minus_reflected(q, z, tau, scz);
    x.Ri[(size_t)x.Np * j + c] = enc2((q.x - to_fix(u.x, 0) + 1) >> 1, (q.y - to_fix(u.y, 0) + 1) >> 1);
    const double2 us = make_double2(u.x * uA, u.y * uA);
    x.row[c] = us;
    if (o == oc + tid) mine = us;
    if (c > i + 1) acc = fma(us.x, us.x, fma(us.y, us.y, acc));
  }
  post_norm(x.nr, acc, oc + (tid & ~31) < ownC, tid >> 5, tid & 31);
  return mine;
}

// x_i (panel column j) and column i+1 of the current matrix for the own rows; its norm
// if it is in the panel.  Returns this thread's first entry of the column.
__device__ __noinline__ double2 finish_column(int i, int j, bool next, int4 ai, int tid) {
  const Ctx &x = ctx();
  const int C = x.C, rank = x.rank, ownR = x.ownR, M = x.M;
  const int o0 = first_own(i + 1, C, rank), kb = (i + 2) & ~31, groups = (ownR - (o0 & ~7) + 31) / 32;
  const int size = row_chunk_size(x.Np - kb, groups), chunks = (x.Np - kb + size - 1) / size;
  const double2 tau = scal(1).tau, scz = scal(1).scz;
  const double uA = pow2(-62);
  const longlong2 *zc = sums(x.zc_at);
  double acc = 0.0;
  double2 mine = make_double2(0.0, 0.0);
  for (int o = o0 + tid; o < ownR; o += kThreads) {
    const int r = glob(o, C, rank);
    if (r >= M) continue;
    if (o != o0 + tid) ai = __ldcg(&x.A[r + (size_t)x.Mp * (i + 1)]);
    longlong2 q = make_longlong2(dec(ai.x, ai.y), dec(ai.z, ai.w)), w = make_longlong2(0, 0);
    for (int ch = 0; ch < chunks; ++ch) {
      const longlong2 t = zc[ch * groups * 32 + o - (o0 & ~7)];
      w.x += t.x;
      w.y += t.y;
    }
    take_off(w, q, ownR, o);
    const double2 a = minus_reflected(q, w, tau, scz);
    x.Li[(size_t)x.Mp * (8 + j) + r] = enc2((q.x - to_fix(a.x, 0) + 1) >> 1, (q.y - to_fix(a.y, 0) + 1) >> 1);
    const double2 as = make_double2(a.x * uA, a.y * uA);
    x.col[r] = as;
    if (o == o0 + tid) mine = as;
    if (r > i + 1) acc = fma(as.x, as.x, fma(as.y, as.y, acc));
  }
  if (next) post_norm(x.nl, acc, o0 + (tid & ~31) < ownR, tid >> 5, tid & 31);
  return mine;
}

// v_i (left; panel column j) of the own rows / u_i of the own columns, from the raw
// vector; mine: this thread's first entry of it
__device__ __noinline__ void put_reflector(bool left, int i, int j, double2 mine, int tid) {
  const Ctx &x = ctx();
  const int C = x.C, rank = x.rank, own = left ? x.ownR : x.ownC, lim = left ? x.M : x.N, one = left ? i : i + 1;
  const double2 sc = scal(left ? 0 : 1).sc;
  const double2 *raw = left ? x.col : x.row;
  int4 *P = left ? x.Li + (size_t)x.Mp * j : x.Ri + (size_t)x.Np * (8 + j);
  int4 *out = left ? reinterpret_cast<int4 *>(x.X) + (size_t)x.M * i : x.Pv + (size_t)x.N * i;
  const int o0 = first_own(one, C, rank) + tid;
  for (int o = o0; o < own; o += kThreads) {
    const int r = glob(o, C, rank);
    if (r >= lim) continue;
    const double2 v = r == one ? make_double2(1.0, 0.0) : cmul(o == o0 ? mine : ldc(&raw[r]), sc);
    P[r] = out[r] = enc2(to_fix(v.x, 62), to_fix(v.y, 62));
  }
  // the back-transformation takes four reflectors together, from the first one's start
  if (x.rank == 0 && tid < (i & 3)) out[one - 1 - tid] = make_int4(8, 0, 8, 0);
}

// raw column q of the matrix (panel start) for the own rows; returns this thread's first entry
__device__ __noinline__ double2 column_start(int q, int tid) {
  const Ctx &x = ctx();
  const int o0 = first_own(q, x.C, x.rank);
  const double uA = pow2(-62);
  double acc = 0.0;
  double2 mine = make_double2(0.0, 0.0);
  for (int o = o0 + tid; o < x.ownR; o += kThreads) {
    const int r = glob(o, x.C, x.rank);
    if (r >= x.M) continue;
    const int4 v = __ldcg(&x.A[r + (size_t)x.Mp * q]);
    const double2 a = make_double2((double)dec(v.x, v.y) * uA, (double)dec(v.z, v.w) * uA);
    x.col[r] = a;
    if (o == o0 + tid) mine = a;
    if (r > q) acc = fma(a.x, a.x, fma(a.y, a.y, acc));
  }
  post_norm(x.nl, acc, o0 + (tid & ~31) < x.ownR, tid >> 5, tid & 31);
  return mine;
}

}  // namespace

__global__ void __launch_bounds__(kThreads, 1) k_gebrd(Slot *slots, const int *path, int keep) {
  namespace cg = cooperative_groups;
  cg::cluster_group cluster = cg::this_cluster();
  const int route = path[blockIdx.y];
  if (!on_route(route)) return;  // uniform per cluster
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const Ctx &x = ctx();
  if (tid == 0) {
    const Slot S = slots[blockIdx.y];
    Ctx &c = ctx();
    bd_dims(*S.cp, route, c.M, c.N);
    c.Mp = up(c.M, 32);
    c.Np = up(c.N, 32);
    c.C = (int)cluster.num_blocks();
    c.rank = (int)cluster.block_rank();
    c.ownR = own_count(c.M, c.C);
    c.ownC = own_count(c.N, c.C);
    c.nnorm = c.C * kWarps;
    c.npb = pair_batch(c.M, c.C);
    c.lf_at = kVec + c.Mp;
    c.zc_at = c.lf_at + 512 * c.npb;
    c.zp_at = c.zc_at + sum_slots(c.M, c.C);
    c.X = S.X;
    c.tau = S.tau;
    c.taup = S.taup;
    c.d = S.bdws;
    c.e = S.bdws + c.N;
    double2 *p = S.aux;
    auto take = [&](size_t n) {
      double2 *q = p;
      p += n;
      return q;
    };
    c.Pv = reinterpret_cast<int4 *>(take((size_t)c.N * c.N));
    c.A = reinterpret_cast<int4 *>(take((size_t)c.Mp * c.Np));
    c.Li = reinterpret_cast<int4 *>(take(16 * (size_t)c.Mp));
    c.Ri = reinterpret_cast<int4 *>(take(16 * (size_t)c.Np));
    c.col = take(c.Mp);
    c.row = take(c.Np);
    c.nl = reinterpret_cast<double *>(take(kWarps / 2 * kMaxC));
    c.nr = reinterpret_cast<double *>(take(kWarps / 2 * kMaxC));
  }
  __syncthreads();
  const int M = x.M, N = x.N;
  // ---- Frobenius norm, scale, fixed-point copy ----
  {
    double acc = 0.0;
    const size_t tot = (size_t)M * N;
    for (size_t e = x.rank * kThreads + tid; e < tot; e += (size_t)x.C * kThreads) {
      const double2 a = x.X[e];
      acc = fma(a.x, a.x, fma(a.y, a.y, acc));
    }
    post_norm(x.nl, acc, true, warp, lane);
    cluster.sync();
    bool fin = true;
    for (int q = lane; q < x.nnorm; q += 32) fin = fin && isfinite(__ldcg(x.nl + q));
    if (!__all_sync(0xffffffffu, fin)) {  // NaN or Inf in Theta: the caller's norm check reports it
      if (x.rank == 0)
        for (int i = tid; i < N; i += kThreads) {
          x.d[i] = nan("");
          if (i < N - 1) x.e[i] = nan("");
          x.tau[i] = x.taup[i] = make_double2(0.0, 0.0);
        }
      return;  // uniform over the cluster: every warp reads the same values
    }
    const int eA = norm_exponent(x.nl, x.nnorm, lane), sh62 = 62 - eA;
    if (tid == 0) ctx().eA = eA;
    const size_t totp = (size_t)x.Mp * x.Np;
    double2 *copy = reinterpret_cast<double2 *>(x.Pv) + bd_theta_at(M, N);
    for (size_t e = x.rank * kThreads + tid; e < totp; e += (size_t)x.C * kThreads) {
      const int r = (int)(e % x.Mp), c = (int)(e / x.Mp);
      double2 a = make_double2(0.0, 0.0);
      if (r < M && c < N) {
        a = x.X[r + (size_t)M * c];
        if (keep) copy[r + (size_t)M * c] = a;
      }
      x.A[e] = enc2(to_fix(a.x, sh62), to_fix(a.y, sh62));
    }
  }
  cluster.sync();
  double2 mine = column_start(0, tid);  // this thread's first own entry of the raw vector
  cluster.sync();
  for (int p = 0; p < N; p += kP) {
    const int jb = min(kP, N - p);
    for (int j = 0; j < jb; ++j) {
      const int i = p + j;
      const bool last = i == N - 1;
      // ================= phase A: left reflector of column i =================
      {
        const int es = norm_exponent(x.nl, x.nnorm, lane);
        if (warp == kWorkers) {
          if (lane < 16) coefficient(x.Li, x.Mp, lane, i, (lane & 7) < j);
          workers_arrive();
          reflector(0, ldc(&x.col[i]), es, i, lane);
        } else {
          if (!last) put_vector(x.col, (i + 1) & ~31, x.Mp, i, M, es, tid);
          workers_sync();
          if (!last) left_products(i, j > 0, warp, lane);
        }
      }
      int4 ai = make_int4(8, 0, 8, 0);  // row i of A0 for the own columns, ahead of its use
      {
        const int c = glob(first_own(i + 1, x.C, x.rank) + tid, x.C, x.rank);
        if (c < N) ai = __ldcg(&x.A[i + (size_t)x.Mp * c]);
      }
      __syncthreads();
      if (last) {
        put_reflector(true, i, j, mine, tid);
        break;
      }
      if (j > 0) {
        if (warp == kWorkers) dots_to_coefficients((lane & 7) < j, lane);  // V^H v, X^H v
        __syncthreads();
        correct(true, i, warp, lane);
        __syncthreads();
      }
      const double2 myrow = finish_row(i, j, ai, tid);
      cluster.barrier_arrive();
      put_reflector(true, i, j, mine, tid);  // the others need it after the next barrier only
      cluster.barrier_wait();
      // ================= phase B: right reflector of row i =================
      {
        const int et = norm_exponent(x.nr, x.nnorm, lane);
        if (warp == kWorkers) {  // y_0..y_j, u_0..u_(j-1) are in use
          if (lane < 16) coefficient(x.Ri, x.Np, lane, i + 1, lane < 8 ? lane <= j : lane - 8 < j);
          workers_arrive();
          reflector(1, ldc(&x.row[i + 1]), et, i, lane);
        } else {
          put_vector(x.row, (i + 2) & ~31, x.Np, i + 1, N, et, tid);
          workers_sync();
          right_products(i, warp, lane);
        }
      }
      ai = make_int4(8, 0, 8, 0);  // column i+1 of A0 for the own rows
      {
        const int r = glob(first_own(i + 1, x.C, x.rank) + tid, x.C, x.rank);
        if (r < M) ai = __ldcg(&x.A[r + (size_t)x.Mp * (i + 1)]);
      }
      __syncthreads();
      if (warp == kWorkers) dots_to_coefficients(lane < 8 ? lane <= j : lane - 8 < j, lane);  // Y^H u, U^H u
      __syncthreads();
      correct(false, i, warp, lane);
      __syncthreads();
      const bool next = j + 1 < jb;
      mine = finish_column(i, j, next, ai, tid);
      if (!next) put_reflector(false, i, j, myrow, tid);  // the panel's end reads it
      cluster.barrier_arrive();
      if (next) put_reflector(false, i, j, myrow, tid);
      cluster.barrier_wait();
    }
    const int q = p + kP;
    if (q >= N) break;
    panel_update(q, warp, lane);
    __syncthreads();
    mine = column_start(q, tid);
    cluster.sync();
  }
}

size_t gebrd_aux_elems(int M, int N) { return bd_theta_at(M, N); }

// k_gebrd on the batch's slots, the largest dimension nmax
int launch_gebrd(tebd_handle *h, const BidiagBatch &b) {
  cudaStream_t st = h->stream;
  const int nb = b.nb, nmax = b.nmax;
  cudaLaunchConfig_t cfg = {};
  cfg.blockDim = dim3(kThreads, 1, 1);
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int rc = check_cuda(h, cudaFuncSetAttribute(k_gebrd, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemMax),
                      "bidiagonalisation shared memory");
  if (rc) return rc;
  // Cluster size: clusters must fit in one GPC, so the co-resident count
  // (occupancy query) decides how many waves a size needs; the time of a batch
  // goes as waves / C for large matrices.
  const int cmax = kMaxC;
  int nbd = 0;  // problems on this route (the others' clusters exit at once)
  for (int s = 0; s < nb; ++s) nbd += b.path_h[s] != kPathQRJ;
  const TuneParams tp = tune_lookup(h, b.dfp ? 1 : 0, nmax, nbd);
  auto co_resident = [&](int c) {
    int ncl = 0;
    cfg.gridDim = dim3(c, nb, 1);
    attr[0].val.clusterDim.x = c;
    cfg.dynamicSmemBytes = smem_bytes(nmax, c);
    if (cfg.dynamicSmemBytes > kSmemMax ||
        cudaOccupancyMaxActiveClusters(&ncl, (const void *)k_gebrd, &cfg) != cudaSuccess) {
      cudaGetLastError();
      ncl = 0;
    }
    return ncl;
  };
  int C = 0;
  double best = 1e300;
  for (int c = 1; c <= cmax; ++c) {
    const int ncl = co_resident(c);
    if (ncl < 1) continue;
    const double cost = (double)((nbd + ncl - 1) / ncl) / c;
    if (cost < best * (1.0 - 1e-9)) {
      best = cost;
      C = c;
    }
  }
  if (tp.cluster > 0) {  // the autotuner's size, when the launch can use it
    if (tp.cluster <= kMaxC && co_resident(tp.cluster) >= 1)
      C = tp.cluster;
    else
      tune_reject(h);
  }
  if (C == 0) return set_error(h, TEBD_ERR_CUDA, "bidiagonalisation: no cluster size fits");
  cfg.gridDim = dim3(C, nb, 1);
  attr[0].val.clusterDim.x = C;
  cfg.dynamicSmemBytes = smem_bytes(nmax, C);
  rc = check_cuda(h, cudaLaunchKernelEx(&cfg, k_gebrd, b.slots_d, b.path_d, (int)!b.right_only),
                  "bidiagonalisation launch");
  TEBD_LAUNCHED(h);
  return rc;
}

}  // namespace tebd
