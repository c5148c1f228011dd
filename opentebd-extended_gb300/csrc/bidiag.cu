// bidiag.cu -- SVD of a large compacted Theta through Householder bidiagonalisation,
// computing only the chi singular triplets the update keeps.
//
// Replaces SVDTruncation's ZGESVD('A','A') (local_operations_module.f90:322-345)
// for bonds of 64 columns or more in a batch that holds a saturated one (where the rank
// approaches n and the QR route's sweeps, O(k^3) each, dominate) or one above 384 columns, and
// for the number-conserving update's blocks of 16 or more.  FormLambda1/FormGamma1/FormGamma2 read
// only the first chi singular values and vectors, so only those are computed:
//   1. (gebrd.cu) ZGEBD2 semantics: Q^H Theta P = B, B real upper bidiagonal (ZLARFG
//      makes beta real), left reflectors H(i) = I - tauq v v^H below the diagonal,
//      right reflectors G(i) = I - taup u u^H (u column-wise in aux).
//   2. Singular values of B: bisection with Sturm counts on the Golub-Kahan
//      tridiagonal (zero diagonal, off-diagonals d0,e0,d1,...,d_{n-1}; its
//      eigenvalues are +-sigma), one thread per kept value, stopped at relative
//      width 2 eps.
//   3. Singular vectors of B: inverse iteration on the Golub-Kahan matrix shifted
//      by sigma_i (tridiagonal LU with partial pivoting, two solves from a fixed
//      start, one more for clusters), eigenvector z = (v0,u0,v1,u1,...)/sqrt2; then (bdorth.cu)
//      the u's and the v's are each re-orthogonalised in descending sigma order.
//   4. (bdapply.cu) U = Q [Ub; 0], V = P Vb by applying the reflectors in reverse, four at
//      a time; X(:,i) = U(:,i) sigma_i, V(:,i), the same layout the sort and restore
//      kernels read from the Jacobi routes.
//   5. (bdrows.cu) small rows of U and V from Theta, to their own size.
// The values and the solves are FP64, everything else 64-bit fixed point, whose products the
// integer pipe does 5 times faster.  Cost: 32/3 n^3 (bidiagonalisation) + 16 (m+n) n chi'
// (back-transformation) instead of the Jacobi route's many O(n k^2) sweeps.
#include <math.h>

#include <algorithm>

#include "bidiag.cuh"
#include "fixed.cuh"

namespace tebd {

namespace {

inline unsigned cdiv(size_t a, size_t b) { return (unsigned)((a + b - 1) / b); }

// limit of the dynamic shared memory, one value for all calls: the attribute belongs to
// the process, and another thread's call may launch in between
constexpr int kSmemMax = 200 * 1024;

}  // namespace

// ---------------------------------------------------------------------------
// 2. bisection: sigma_i of B for i < kk (one team of kTeam lanes each), Golub-Kahan Sturm counts
// ---------------------------------------------------------------------------
// Sturm counts of the Golub-Kahan matrix (eigenvalues below x) from the characteristic
// polynomials of its leading blocks, p_{j+2} = -x p_{j+1} - o_j^2 p_j: the count is the number
// of sign changes, a zero counting as either sign.  No divisions: an FP64 step is two
// instructions (130 cycles of a scheduler) where the quotient form's takes 645, and one
// FP32 step 10 cycles against 45.  Each computed p_{j+2} satisfies the recurrence with x and
// o_j^2 changed by a few ulps, so that the counts are those of a matrix that close, as
// the quotient form's.  Everything is scaled by the Gershgorin bound (entries in [0, 1]),
// and the pair is rescaled by powers of two every kRescale steps; squared off-diagonals
// below kTiny2 (kTiny2F) are raised to it, far below what a count resolves, so that the
// pair cannot vanish in between.
constexpr int kRescale = 8, kRescaleF = 4;
constexpr double kTiny2 = 1e-70;
constexpr float kTiny2F = 1e-14f;

__device__ __forceinline__ int gk_count(const double *sq, int n1, double x) {
  double p0 = 1.0, p1 = -x;
  int c = 1;  // x > 0
  for (int j = 0; j < n1; j += kRescale) {
#pragma unroll
    for (int u = 0; u < kRescale; ++u)
      if (j + u < n1) {
        const double p2 = fma(-x, p1, -sq[j + u] * p0);
        c += (unsigned)(__double2hiint(p2) ^ __double2hiint(p1)) >> 31;
        p0 = p1;
        p1 = p2;
      }
    const int e = (max(__double2hiint(p0) & 0x7fffffff, __double2hiint(p1) & 0x7fffffff) >> 20) - 1023;
    if (e != 0) {  // both by 2^-e (what underflows is far below the other)
      const int h0 = __double2hiint(p0), h1 = __double2hiint(p1), sh = e << 20;
      p0 = (h0 & 0x7ff00000) > max(sh, 0) ? __hiloint2double(h0 - sh, __double2loint(p0)) : copysign(0.0, p0);
      p1 = (h1 & 0x7ff00000) > max(sh, 0) ? __hiloint2double(h1 - sh, __double2loint(p1)) : copysign(0.0, p1);
    }
  }
  return c;
}

__device__ __forceinline__ int gk_count_f32(const float *sqf, int n1, float x) {
  float p0 = 1.0f, p1 = -x;
  int c = 1;
  for (int j = 0; j < n1; j += kRescaleF) {
#pragma unroll
    for (int u = 0; u < kRescaleF; ++u)
      if (j + u < n1) {
        const float p2 = fmaf(-x, p1, -sqf[j + u] * p0);
        c += (unsigned)(__float_as_int(p2) ^ __float_as_int(p1)) >> 31;
        p0 = p1;
        p1 = p2;
      }
    const int e = max(__float_as_int(p0) & 0x7fffffff, __float_as_int(p1) & 0x7fffffff) >> 23;
    const float s = __int_as_float(max(1, min(253, 254 - e)) << 23);  // about 2^-(e - 127)
    p0 *= s;
    p1 *= s;
  }
  return c;
}

// sigma_i of B for i < min(kk, n), descending.
//   1. FP32 bisection on the scaled problem to width 2^-22 ||T||; FP32 counts are exact
//      for a T perturbed by a few float ulps, so the bracket widened by 2^-18 ||T|| holds
//      sigma_i; two FP64 counts check it (reset to [0, ||T||] otherwise).
//   2. FP64 bisection to width 2 eps sigma + eps ||T||: the absolute accuracy LAPACK's
//      bidiagonal SVD reaches on Theta as a whole.
// Each value is found by a team of kTeam lanes that evaluate kTeam points of the bracket
// at once (multisection): the counts are monotone in x, so the leading run of "count <=
// target" in the team's ballot picks one of kTeam + 1 subintervals (16 lanes: 4.1 bits per
// step instead of bisection's 1).  While the values leave schedulers idle, the
// sequential recurrences bound the kernel and extra lanes are free; once there is a warp
// per scheduler, teams of 1 lane (bisection) do the least work.  The host picks kTeam
// per launch; where sizes differ a value counts by its problem's share of the largest (its
// lanes are free that much earlier).  Measured: 128 values of 32 bonds, n = 640: 7.8 -> 2.4 ms; 90 of 10, n =
// 270: 2.26 -> 0.60 ms.
constexpr int kSigmaThreads = 32;
template <int kTeam>
__global__ void __launch_bounds__(kSigmaThreads) k_bd_sigma(Slot *slots, const int *path, int kk) {
  constexpr int kSigmaValues = kSigmaThreads / kTeam;  // values per block
  // step cap (safety only; the width test ends the loop): log2(kTeam + 1) bits per step
  constexpr int kIt32 = kTeam == 1 ? 26 : kTeam == 2 ? 17 : kTeam == 4 ? 12 : 10;
  const int s = blockIdx.y;
  const int route = path[s];
  if (!on_route(route)) return;
  const Slot S = slots[s];
  int m, n;
  bd_dims(*S.cp, route, m, n);
  const int K = min(kk, n);
  if ((int)(blockIdx.x * kSigmaValues) >= K) return;  // uniform per block
  const int n1 = 2 * n - 1;
  extern __shared__ double sq[];  // n1 scaled squared off-diagonals, then in FP32
  float *sqf = reinterpret_cast<float *>(sq + n1);
  const double *dd = S.bdws, *ee = S.bdws + n;
  double hl = 0.0;
  for (int j = threadIdx.x; j < n; j += blockDim.x)
    hl = fmax(hl, fabs(dd[j]) + (j < n - 1 ? fabs(ee[j]) : 0.0) + (j > 0 ? fabs(ee[j - 1]) : 0.0));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) hl = fmax(hl, __shfl_xor_sync(0xffffffffu, hl, o));
  const double hi = hl * (1.0 + 1e-12) + 1e-300;  // Gershgorin bound of the Golub-Kahan matrix
  const double inv_hi = 1.0 / hi;
  for (int j = threadIdx.x; j < n1; j += blockDim.x) {
    const double o = (j & 1) ? ee[j >> 1] : dd[j >> 1];
    const double os = (o * inv_hi) * (o * inv_hi);
    sq[j] = os < kTiny2 ? kTiny2 : os;
    sqf[j] = fmaxf((float)os, kTiny2F);
  }
  __syncthreads();
  const int team = threadIdx.x / kTeam, t = threadIdx.x % kTeam;
  const unsigned tmask = (kTeam == 32 ? 0xffffffffu : ((1u << kTeam) - 1u)) << (kTeam * team);
  const int i = blockIdx.x * kSigmaValues + team;
  if (i >= K) return;  // the whole team leaves together
  const int target = 2 * n - 1 - i;  // count(< x) <= target  <=>  x <= sigma_i
  // leading run of true votes of the team (bit t: point t has count <= target)
  auto lead = [&](bool ok) -> int {
    const unsigned b = (__ballot_sync(tmask, ok) & tmask) >> (kTeam * team);
    return b == (kTeam == 32 ? 0xffffffffu : (1u << kTeam) - 1u) ? kTeam : __ffs(~b) - 1;
  };
  // 1. FP32 bracket of width 2^-22
  float lf = 0.0f, hf = 1.0f;
  for (int it = 0; it < kIt32 && hf - lf > 2.384185791015625e-07f; ++it) {
    const float w = (hf - lf) * (1.0f / (kTeam + 1));
    const int k = lead(gk_count_f32(sqf, n1, lf + w * (float)(t + 1)) <= target);
    const float nl = k > 0 ? lf + w * (float)k : lf;
    hf = k < kTeam ? lf + w * (float)(k + 1) : hf;
    lf = nl;
  }
  // widened by 2^-18, and checked
  double lo = fmax(0.0, (double)lf - 3.814697265625e-06), h = fmin(1.0, (double)hf + 3.814697265625e-06);
  bool good;
  if (kTeam == 1) {
    good = (lo <= 0.0 || gk_count(sq, n1, lo) <= target) && gk_count(sq, n1, h) > target;
  } else {
    const int c = gk_count(sq, n1, t == 0 ? fmax(lo, 1e-300) : h);
    good = __all_sync(tmask, t > 1 || (t == 0 ? c <= target : c > target));
  }
  if (!good) {
    lo = 0.0;
    h = 1.0;
  }
  // 2. FP64 multisection to 2 eps sigma + eps ||T||
  for (int it = 0; it < 80; ++it) {
    if (h - lo <= 4.440892098500626e-16 * h + 2.220446049250313e-16 || h < 1e-30) break;
    const double w = (h - lo) * (1.0 / (kTeam + 1));
    const int k = lead(gk_count(sq, n1, lo + w * (double)(t + 1)) <= target);
    const double nl = k > 0 ? lo + w * (double)k : lo;
    h = k < kTeam ? lo + w * (double)(k + 1) : h;
    lo = nl;
  }
  const double sg = 0.5 * (lo + h);
  if (t == 0) S.bdws[2 * n + i] = sg < 1e-30 ? 0.0 : sg * hi;
}

// ---------------------------------------------------------------------------
// 3a. inverse iteration on (T_GK - sigma_i I), one thread per value: two solves.  Inside a
// cluster the raw vectors are combinations of the cluster's, the same ones of the v's and of
// the u's, but each set is re-orthogonalised by itself, and the two agree only to eps
// times the raw vectors' condition (1e5 and more where rounding spreads a cluster over the
// distance of the shift).  Problems with values within 64 ulps of the next
// (bd_clustered) go through a second pass, one solve from the orthogonal vectors and the
// re-orthogonalisation again, whose raw vectors are nearly orthogonal.  Theta rebuilt,
// relative to its norm, before (rows of a cosine transform as starts, one pass) and now: 64
// values in multiplets of 2 to 21, up to 1.5e-12 -> 5e-15; 256 equal values, 9e-13 -> 4e-14 and
// in the double-float form 2e-8 -> 8e-14.
// Scratch per value (transposed so that threads of a warp touch adjacent words):
//   U0 (reciprocal pivots), U1, U2 (upper factor of the pivoted LU), PV (multipliers),
//   Y (swap flags, ints), then the vector Z itself.
// ---------------------------------------------------------------------------
// An FP64 instruction holds its scheduler for 65 cycles here and a batch has about a warp
// per scheduler, so the loops keep to the few that the solves need (comparisons, row
// swaps and power-of-two scaling on the integer pipe) and load kAhead steps' entries
// before they are used.  Measured: 128 values of 32 bonds, n = 640: 6.4 -> 2.5 ms; 90 of
// 10, n = 270: 1.77 -> 0.92 ms.
constexpr int kAhead = 8;
__device__ __forceinline__ unsigned long long abs_bits(double x) {
  return (unsigned long long)__double_as_longlong(x) & 0x7fffffffffffffffull;
}
__device__ __forceinline__ double times_pow2(double x, int e) {  // x 2^e; 0 where it underflows
  const int h = __double2hiint(x), f = ((h >> 20) & 0x7ff) + e;
  return f <= 0 || (h & 0x7ff00000) == 0 ? 0.0 : __hiloint2double(h + (e << 20), __double2loint(x));
}
__global__ void __launch_bounds__(32) k_bd_invit(Slot *slots, const int *path, int kk, int cap, int second) {
  const int s = blockIdx.y;
  const int route = path[s];
  if (!on_route(route)) return;
  const Slot S = slots[s];
  int m, n;
  bd_dims(*S.cp, route, m, n);
  const int N = 2 * n;
  const int K = cap ? min(min(kk, n), S.cp->k) : min(kk, n);
  if ((int)(blockIdx.x * blockDim.x) >= K) return;  // uniform
  const int i = min((int)(blockIdx.x * blockDim.x + threadIdx.x), K - 1);
  const bool mine = (int)(blockIdx.x * blockDim.x + threadIdx.x) < K;
  const double *dd = S.bdws, *ee = S.bdws + n, *sig = S.bdws + 2 * n;
  if (second && !bd_clustered(sig, K)) return;  // uniform
  double *base = S.bdws + bd_scratch(n, kk);
  double *U0 = base, *U1 = base + (size_t)N * K, *U2 = base + 2 * (size_t)N * K, *PV = base + 3 * (size_t)N * K,
         *Z = base + 5 * (size_t)N * K;
  int *Y = reinterpret_cast<int *>(base + 4 * (size_t)N * K);  // 1: rows j and j + 1 swapped
#define AT(A, j) A[(size_t)(j) * K + i]
  extern __shared__ double off[];  // T(j, j+1), j < N - 1
  for (int j = threadIdx.x; j < N - 1; j += 32) off[j] = (j & 1) ? ee[j >> 1] : dd[j >> 1];
  __syncwarp();
  // pivots below eps ||T|| are raised to it (sign kept), as LAPACK's DLAGTS does,
  // so the solve stays finite when sigma_i is an eigenvalue to working precision
  unsigned long long tb = 0;
  for (int j = threadIdx.x; j < N - 1; j += 32) tb = max(tb, abs_bits(off[j]));
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) tb = max(tb, __shfl_xor_sync(0xffffffffu, tb, o));
  if (!mine) return;
  double lam = sig[i];
  // an exactly zero value: FormLambda1 drops it, its vectors are zero; neither are there vectors
  // of a non-finite B (reported by the norm check), whose solves would rescale at every step
  if (lam <= 0.0 || tb >= 0x7ff0000000000000ull) {
    for (int j = 0; j < N; ++j) AT(Z, j) = 0.0;
    return;
  }
  const double ptol = fmax(2.220446049250313e-16 * __longlong_as_double((long long)tb), 1e-300);
  // Inside a cluster (values within 8 ulps of the largest of one another; the bisection and the
  // rounding of B spread a degenerate value that far) the shift lies 64 ulps above the value,
  // so that the members are all about as far from it and the solves leave each a like share
  // of the cluster's vectors.  With the value itself as the shift one member takes all: the
  // set's condition is 1e6 to 1e13, and its left and right vectors, each re-orthogonalised,
  // no longer belong together (Theta rebuilt from 64 equal values was off by 8e-10 of its
  // norm).  It stays at a quarter of the way to the next value above the cluster, which would
  // take over otherwise, and at 1/64 of the value, whose negative is an eigenvalue
  // too: with 64 ulps everywhere the left and right vectors of values below 1e-14 of the
  // largest were paired at random.  Other values are the shift themselves: a neighbour at a
  // distance g leaves a share of (ulp / g)^2, which costs Theta that share of g.
  // The second pass (below) starts from orthogonal vectors: one solve, 16 ulps above.
  {
    const double ulp = 2.220446049250313e-16 * sig[0], near = 8.0 * ulp, own = lam;
    if (second) {
      lam = own + fmin(16.0 * ulp, 0.015625 * own);
    } else if ((i > 0 && sig[i - 1] - own <= near) || (i + 1 < K && own - sig[i + 1] <= near)) {
      int j = i;  // the cluster's first value
      while (j > 0 && sig[j - 1] - sig[j] <= near) --j;
      double shift = fmin(64.0 * ulp, 0.015625 * own);
      if (j > 0) shift = fmin(shift, 0.25 * (sig[j - 1] - own));
      lam = own + shift;
    }
  }
  const unsigned long long pbits = abs_bits(ptol);
  auto guard = [&](double p) -> double { return abs_bits(p) >= pbits ? p : copysign(ptol, p); };
  // LU with partial pivoting of T - lam I (diagonal -lam, off-diagonals off[j])
  double d0 = -lam, d1 = N > 1 ? off[0] : 0.0;
  for (int j = 0; j < N - 1; ++j) {
    const double sb = off[j], nd0 = -lam, nd1 = j + 1 < N - 1 ? off[j + 1] : 0.0;
    const bool keep = abs_bits(d0) >= abs_bits(sb);  // row j stays the pivot row
    const double rp = 1.0 / (keep ? guard(d0) : sb), mult = (keep ? sb : d0) * rp;
    const double up = keep ? d1 : nd0;
    AT(U0, j) = rp;
    AT(U1, j) = up;
    AT(U2, j) = keep ? 0.0 : nd1;
    AT(PV, j) = mult;
    AT(Y, j) = keep ? 0 : 1;
    d0 = fma(-mult, up, keep ? nd0 : d1);
    d1 = keep ? nd1 : -mult * nd1;
  }
  AT(U0, N - 1) = 1.0 / guard(d0);  // U0 holds the reciprocal pivots
  // start vector: pseudo-random entries in [-1, 1), independent for each value i and entry
  // j (a published integer hash, Wellons' lowbias32, of both).  The vectors of a multiplet
  // are local in B, and over a short window the starts have to be independent too:
  // rows of a cosine transform with common signs are nearly parallel there.
  for (int j = 0; j < N && !second; ++j) {
    unsigned x = ((unsigned)j * 0x9E3779B9u) ^ ((unsigned)(i + 1) * 0x85EBCA6Bu);
    x ^= x >> 16;
    x *= 0x7feb352du;
    x ^= x >> 15;
    x *= 0x846ca68bu;
    x ^= x >> 16;
    AT(Z, j) = (double)(int)x * 4.656612873077393e-10;
  }
  int scale = 0;  // the right-hand side is Z 2^scale
  for (int it = 0; it < (second ? 1 : 2); ++it) {
    // forward: the row operations (with swaps) applied to the right-hand side
    double carry = times_pow2(AT(Z, 0), scale);
    for (int j = 0; j < N - 1; j += kAhead) {
      double z[kAhead], pv[kAhead];
      int sw[kAhead];
#pragma unroll
      for (int u = 0; u < kAhead; ++u)
        if (j + u < N - 1) {
          z[u] = AT(Z, j + u + 1);
          pv[u] = AT(PV, j + u);
          sw[u] = AT(Y, j + u);
        }
#pragma unroll
      for (int u = 0; u < kAhead; ++u)
        if (j + u < N - 1) {
          const double next = times_pow2(z[u], scale);
          AT(Z, j + u) = sw[u] ? next : carry;
          carry = fma(-pv[u], sw[u] ? next : carry, sw[u] ? carry : next);
        }
    }
    AT(Z, N - 1) = carry;
    // back substitution with the upper factor (diagonal U0, super-diagonals U1, U2);
    // a partial result that grows past 2^500 is rescaled, with the values already
    // produced and the right-hand side, so that nothing overflows
    double x1 = 0.0, x2 = 0.0;
    int top = 0;  // largest exponent field
    for (int j = N - 1; j >= 0; j -= kAhead) {
      double z[kAhead], u0[kAhead], u1[kAhead], u2[kAhead];
#pragma unroll
      for (int u = 0; u < kAhead; ++u)
        if (j - u >= 0) {
          z[u] = AT(Z, j - u);
          u0[u] = AT(U0, j - u);
          u1[u] = j - u + 1 < N ? AT(U1, j - u) : 0.0;
          u2[u] = j - u + 2 < N ? AT(U2, j - u) : 0.0;
        }
#pragma unroll
      for (int u = 0; u < kAhead; ++u)
        if (j - u >= 0) {
          double x = fma(-u2[u], x2, fma(-u1[u], x1, z[u])) * u0[u];
          int f = (__double2hiint(x) >> 20) & 0x7ff;
          if (f > 1023 + 500 && f != 0x7ff) {
            for (int q = j - u + 1; q < N; ++q) AT(Z, q) = times_pow2(AT(Z, q), -500);
            for (int q = 0; q < j - u; ++q) AT(Z, q) = times_pow2(AT(Z, q), -500);
#pragma unroll
            for (int v = 0; v < kAhead; ++v)
              if (v > u) z[v] = times_pow2(z[v], -500);
            x = times_pow2(x, -500);
            x1 = times_pow2(x1, -500);
            f -= 500;
            top -= 500;
          }
          AT(Z, j - u) = x;
          top = max(top, f);
          x2 = x1;
          x1 = x;
        }
    }
    scale = 1023 - top;
  }
  double nrm = 0.0;
  for (int j = 0; j < N; j += kAhead) {
    double z[kAhead];
#pragma unroll
    for (int u = 0; u < kAhead; ++u) z[u] = j + u < N ? AT(Z, j + u) : 0.0;
#pragma unroll
    for (int u = 0; u < kAhead; ++u) {
      z[u] = times_pow2(z[u], scale);
      nrm = fma(z[u], z[u], nrm);
    }
  }
  const double inv = nrm > 0.0 ? 1.0 / sqrt(nrm) : 0.0;
  for (int j = 0; j < N; j += kAhead) {
    double z[kAhead];
#pragma unroll
    for (int u = 0; u < kAhead; ++u) z[u] = j + u < N ? AT(Z, j + u) : 0.0;
#pragma unroll
    for (int u = 0; u < kAhead; ++u)
      if (j + u < N) AT(Z, j + u) = times_pow2(z[u], scale) * inv;
  }
#undef AT
}

// the orthogonal vectors (bdorth.cu) back into z, the starts of the second pass
__global__ void __launch_bounds__(256) k_bd_zback(Slot *slots, const int *path, int kk, int cap) {
  __shared__ double tile[2][32][33];
  const int s = blockIdx.z;
  const int route = path[s];
  if (!on_route(route)) return;
  const Slot S = slots[s];
  int m, n;
  bd_dims(*S.cp, route, m, n);
  const int K = cap ? min(min(kk, n), S.cp->k) : min(kk, n);
  const int i0 = blockIdx.x * 32, j0 = blockIdx.y * 32;
  if (i0 >= K || j0 >= n || !bd_clustered(S.bdws + 2 * n, K)) return;  // uniform
  double *base = S.bdws + bd_scratch(n, kk), *Z = base + 5 * (size_t)(2 * n) * K;
  const int2 *Zi = reinterpret_cast<const int2 *>(base);
  const double unit = 2.168404344971009e-19;  // 2^-62
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  for (int y = ty; y < 64; y += 8) {
    const int p = y >> 5, i = i0 + (y & 31), j = j0 + tx;
    if (j < n && i < K) {
      const int2 z = Zi[((size_t)p * K + i) * n + j];
      tile[p][tx][y & 31] = (double)dec(z.x, z.y) * unit;
    }
  }
  __syncthreads();
  for (int y = ty; y < 64; y += 8) {
    const int j = j0 + (y >> 1), i = i0 + tx;
    if (j < n && i < K) Z[(size_t)(2 * j + (y & 1)) * K + i] = tile[y & 1][y >> 1][tx];
  }
}

// 3b. the v's (even rows) and u's (odd rows) re-orthogonalised: bdorth.cu
// 4. left vectors Q [Ub; 0] (M x K) and right vectors P Vb (N x K): bdapply.cu

// X(:, i) = U(:, i) sigma_i (Theta's m rows, ld m) and, on the transposed route,
// V(:, i) = the left vectors of Theta^H (n rows, ld n).
__global__ void k_bd_store(Slot *slots, const int *path, int kk, int cap, int right_only) {
  const int s = blockIdx.y;
  const int route = path[s];
  if (!on_route(route)) return;
  const Slot S = slots[s];
  int M, N;
  bd_dims(*S.cp, route, M, N);
  const int m = S.cp->m, n = S.cp->n, K = cap ? min(min(kk, N), S.cp->k) : min(kk, N);
  double *base = S.bdws + bd_scratch(N, kk);
  const double *sig = S.bdws + 2 * N;
  const double2 *Yu = reinterpret_cast<const double2 *>(base + 12 * (size_t)N * K);
  const double2 *U = route == kPathBidiagT ? reinterpret_cast<const double2 *>(base + 10 * (size_t)N * K) : Yu;
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; !right_only && e < (size_t)m * K; e += stride) {
    const int i = (int)(e / m);
    const double2 y = U[e];
    S.X[e] = make_double2(y.x * sig[i], y.y * sig[i]);
  }
  if (route == kPathBidiagT)
    for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < (size_t)n * K; e += stride)
      S.V[e] = Yu[e];
  if (cap) {  // columns past the capped count read as zero singular values
    for (size_t e = (size_t)m * K + blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < (size_t)m * n; e += stride)
      S.X[e] = make_double2(0.0, 0.0);
  } else if (blockIdx.x == 0 && threadIdx.x == 0) {
    S.cp->k = K;
  }
}

// Transposed route, before the bidiagonalisation: X (m x n, ld m) -> V (copy),
// then X <- V^H (n x m, ld n).
__global__ void k_bd_stage(Slot *slots, const int *path) {
  const int s = blockIdx.y;
  if (path[s] != kPathBidiagT) return;
  const Slot S = slots[s];
  const size_t e_end = (size_t)S.cp->m * S.cp->n;
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < e_end;
       e += (size_t)gridDim.x * blockDim.x)
    S.V[e] = S.X[e];
}

__global__ void k_bd_transpose(Slot *slots, const int *path) {
  __shared__ double2 tile[32][33];
  const int s = blockIdx.z;
  if (path[s] != kPathBidiagT) return;
  const Slot S = slots[s];
  const int m = S.cp->m, n = S.cp->n;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;  // 32 x 8 threads
  for (int tr = blockIdx.y * 32; tr < m; tr += gridDim.y * 32)
    for (int tc = blockIdx.x * 32; tc < n; tc += gridDim.x * 32) {
      for (int q = ty; q < 32; q += 8) {  // read V(tr + tx, tc + q)
        const int r = tr + tx, c = tc + q;
        if (r < m && c < n) tile[q][tx] = S.V[r + (size_t)m * c];
      }
      __syncthreads();
      for (int q = ty; q < 32; q += 8) {  // write X(tc + tx, tr + q) = conj(V(tr + q, tc + tx))
        const int c = tc + tx, r = tr + q;
        if (r < m && c < n) {
          const double2 v = tile[tx][q];
          S.X[c + (size_t)n * r] = make_double2(v.x, -v.y);
        }
      }
      __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// host orchestration: bidiagonal route for the slots flagged kPathBidiag / kPathBidiagT
// ---------------------------------------------------------------------------
size_t bidiag_aux_elems(int n) { return gebrd_aux_elems(n, n) + bd_rows_aux_elems(n, n); }

size_t bidiag_ws_doubles(int n, int chi) {
  const int K = std::min(chi, n);
  return bd_scratch(n, chi) + 6 * (size_t)(2 * n) * K + 2 * (size_t)n * K + bd_orth_ws_doubles(K);
}

int run_bidiag_batch(tebd_handle *h, const BidiagBatch &b) {
  cudaStream_t st = h->stream;
  const int kk = b.kk, nb = b.nb, nmax = b.nmax, cap = b.cap;
  Slot *slots_d = b.slots_d;
  const int *path_d = b.path_d;
  int rc;
  if (b.phase != 2) {  // bidiagonalisation and singular values
  if (h->profiling) cudaEventRecord(h->ev[0], st);
  bool any_t = false;
  for (int s = 0; s < nb; ++s) any_t |= b.path_h[s] == kPathBidiagT;
  if (any_t) {
    k_bd_stage<<<dim3(128, nb), 256, 0, st>>>(slots_d, path_d);
    TEBD_LAUNCHED(h);
    const unsigned g = cdiv(nmax, 32) < 8 ? cdiv(nmax, 32) : 8;
    k_bd_transpose<<<dim3(g, g, nb), 256, 0, st>>>(slots_d, path_d);
    TEBD_LAUNCHED(h);
  }
  if (h->profiling) cudaEventRecord(h->ev[4], st);
  if ((rc = launch_gebrd(h, b))) return rc;
  if (h->profiling) cudaEventRecord(h->ev[5], st);
  ++h->stats.gebrd_launches;
  {
    const size_t smem = (sizeof(double) + sizeof(float)) * (size_t)(2 * nmax);
    // team size: multisection while the batch's values (nb x kk at most) leave warp
    // schedulers idle, plain bisection once there is a warp for each
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const double values = b.values > 0 ? b.values : (double)nb * std::min(kk, nmax), lanes = 4.0 * 32.0 * std::max(sms, 1);
    int team = 1;
    while (team < 16 && values * 2 * team <= lanes) team *= 2;
    const TuneParams tp = tune_lookup(h, b.dfp ? 1 : 0, nmax, nb);
    if (tp.team == 1 || tp.team == 2 || tp.team == 4 || tp.team == 8) team = tp.team;
    auto kern = team == 16  ? k_bd_sigma<16>
                : team == 8 ? k_bd_sigma<8>
                : team == 4 ? k_bd_sigma<4>
                : team == 2 ? k_bd_sigma<2>
                            : k_bd_sigma<1>;
    if ((rc = check_cuda(h, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax),
                         "bisection shared memory")))
      return rc;
    kern<<<dim3(cdiv(kk, kSigmaThreads / team), nb), kSigmaThreads, smem, st>>>(slots_d, path_d, kk);
  }
  TEBD_LAUNCHED(h);
  if (b.phase == 1) return check_cuda(h, cudaGetLastError(), "bidiag launch");
  }  // vectors
  {
    const size_t smem = sizeof(double) * (size_t)(2 * nmax);
    if ((rc = check_cuda(h, cudaFuncSetAttribute(k_bd_invit, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemMax),
                         "inverse iteration shared memory")))
      return rc;
    int clusters = 0;  // of k_bd_orth, the same in both passes
    for (int second = 0; second < (b.right_only ? 1 : 2); ++second) {  // the second: problems with clustered values
      if (second) {
        k_bd_zback<<<dim3(cdiv(kk, 32), cdiv(nmax, 32), nb), 256, 0, st>>>(slots_d, path_d, kk, cap);
        TEBD_LAUNCHED(h);
      }
      k_bd_invit<<<dim3(cdiv(kk, 32), nb), 32, smem, st>>>(slots_d, path_d, kk, cap, second);
      TEBD_LAUNCHED(h);
      if ((rc = launch_bd_orth(h, b, second, &clusters))) return rc;
    }
  }
  if ((rc = launch_bd_apply(h, b))) return rc;
  if (!b.right_only && (rc = launch_bd_rows(h, b))) return rc;
  k_bd_store<<<dim3(256, nb), 256, 0, st>>>(slots_d, path_d, kk, cap, b.right_only);
  TEBD_LAUNCHED(h);
  if (h->profiling) {
    cudaEventRecord(h->ev[1], st);
    if ((rc = check_cuda(h, cudaStreamSynchronize(st), "bidiag"))) return rc;
    float ms = 0.f;
    if (cudaEventElapsedTime(&ms, h->ev[0], h->ev[1]) == cudaSuccess) h->stats.bidiag_ms += ms;
    if (cudaEventElapsedTime(&ms, h->ev[4], h->ev[5]) == cudaSuccess) h->stats.gebrd_ms += ms;
  }
  return check_cuda(h, cudaGetLastError(), "bidiag launch");
}

int run_bidiag(tebd_handle *h, int nb, int nmax) {
  BidiagBatch b;
  b.slots_d = h->slots_d;
  b.path_d = h->path_d;
  b.path_h = h->path_h.data();
  b.nb = nb;
  b.nmax = nmax;
  b.kk = h->chi;
  // the precision form, and the learned-rank form's bonds off the randomized route
  b.dfp = h->opts.svd_mode == TEBD_SVD_DF || h->opts.svd_mode == TEBD_SVD_RSVD;
  b.phase = 0;
  b.cap = 0;
  return run_bidiag_batch(h, b);
}

// Workspace of one bidiagonal problem of M x N (M >= N) computing all N triplets
// (kk = the batch's largest N): aux, tau, taup (complex) and bdws (doubles).
void bidiag_block_ws(int M, int N, int kk, size_t *aux_elems, size_t *bdws_doubles) {
  const int K = std::min(kk, N);
  *aux_elems = gebrd_aux_elems(M, N) + bd_rows_aux_elems(M, N);
  *bdws_doubles = bd_scratch(N, kk) + 6 * (size_t)(2 * N) * K + 2 * (size_t)M * K + bd_orth_ws_doubles(K) + 4;
}

}  // namespace tebd
