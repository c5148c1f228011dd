// qrj.cu -- SVD of the compacted Theta by rank-revealing QR + one-sided Jacobi.
//
// Replaces SVDTruncation's ZGESVD('A','A') (local_operations_module.f90:322-345)
// for the dense update of an unsaturated bond.  The algorithm is the preconditioned
// Jacobi SVD of Drmac and Veselic (the method behind LAPACK's xGEJSV):
//   1. Householder QR with column pivoting, Theta P = Q R (ZGEQP3 semantics: largest
//      remaining column first, column-norm downdating with recomputation on
//      cancellation), stopped at the numerical rank k: the first step whose largest
//      remaining column norm is below 2^-60 ||Theta||_F.  The neglected block has norm
//      <= sqrt(n) 2^-60 ||Theta||, three decades under the reference's 1e-15 Lambda guard.
//   2. A second QR, R^H = Q2 R2, so that the sweeps work on k x k instead of n x k.
//   3. One-sided Jacobi on X = R2^H (lower triangular, graded): X Z = W Sigma in a few
//      sweeps.
//   4. Theta = (Q W) Sigma (P Q2 Z)^H: the reflectors applied to W Sigma and to Z.
// Every step is FP64.  The work is O(m n k) for the QRs and O(k^3) per sweep, and k is
// the Schmidt rank of the bond, which is far below d*chi until the chain saturates.
//
// The FP64 pipes bound the QR (an instruction of a warp takes its scheduler 65 cycles),
// so its kernel spends them on the products only: a cluster of CTAs per bond with the
// columns dealt out to them in shared memory, squared norms instead of norms, unscaled
// reflectors (one square root and one quotient per step, where the norm of every column
// took two of each), and one cluster barrier per step: every CTA finds the pivot and
// forms the reflector by itself.
//
// Measured: 24 batches of 32 bonds, rank about 36 of 160 columns: both QRs 70 -> 21.8 ms, the
// sweeps 105 -> 73.6 ms; 36 batches of 16, rank 10 of 20: 7.4 -> 4.3 and 10 -> 7.0 ms.
#include <cooperative_groups.h>
#include <math.h>

#include <algorithm>

#include "tebd_internal.cuh"

namespace tebd {

int jacobi_persistent_double(tebd_handle *h, const JacobiProblem<double> *probs_d, int nprob,
                             int nmax, double tol, int max_sweeps);

namespace {
namespace cg = cooperative_groups;

constexpr int kQW = 16, kQThreads = 32 * kQW;  // of the QR kernel
constexpr int kMaxC = 8;
constexpr size_t kSmemMax = 220 * 1024;

__device__ __forceinline__ double wsum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
// two sums over the lanes, in every lane
__device__ __forceinline__ void wsum2(double &a, double &b, int lane) {
  const bool up = lane & 16;
  double x = (up ? b : a) + __shfl_xor_sync(0xffffffffu, up ? a : b, 16);
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  a = __shfl_sync(0xffffffffu, x, 0);
  b = __shfl_sync(0xffffffffu, x, 16);
}
__device__ __forceinline__ double pow2(int e) { return __hiloint2double((e + 1023) << 20, 0); }

__host__ __device__ __forceinline__ size_t qr_scratch(int mx) { return (56 * (size_t)mx + 15) & ~(size_t)15; }  // bytes per CTA
__host__ __device__ __forceinline__ size_t qr_columns(int mx, int C) {
  return 16 * (size_t)mx * ((mx + C - 1) / C);
}

// One factorisation by a cluster.  Scratch of a CTA (shared memory, or global for a
// matrix that it cannot hold): the reflector, squared norms (remaining, before odd and even
// steps, so that a CTA may be a step's search behind; and at their last computation), diagonal of R, position -> column and column -> position.
struct Qr {
  int M, N, C, rank;
  double2 *own;   // this CTA's columns (shared memory), null: in `glob`
  double2 *glob;  // the matrix, ld M
  double2 *v;
  double *n1[2], *n2, *beta;
  int *perm, *pos;
  char *scr;      // global scratch of CTA 0, null: shared memory
  size_t stride;
  __device__ __forceinline__ double2 *column(int c) const {
    return own ? own + (size_t)(c / C) * M : glob + (size_t)M * c;
  }
  // CTA r's copy of a scratch entry
  __device__ __forceinline__ double *of(cg::cluster_group &cluster, double *p, int r) const {
    if (!scr) return cluster.map_shared_rank(p, r);
    return reinterpret_cast<double *>(reinterpret_cast<char *>(p) + ((long long)r - rank) * (long long)stride);
  }
  __device__ __forceinline__ void place(char *p, int mx) {
    v = reinterpret_cast<double2 *>(p);
    n1[0] = reinterpret_cast<double *>(v + mx);
    n1[1] = n1[0] + mx;
    n2 = n1[1] + mx;
    beta = n2 + mx;
    perm = reinterpret_cast<int *>(beta + mx);
    pos = perm + mx;
  }
};

// Steps 0 .. kmax - 1, until the largest remaining column is at most sqrt(tol2) (kPivot).
// Reflector j, unscaled (H^H = I - t v v^H with v_j = alpha - beta, t = -1 / (beta v_j)),
// goes to QV(:, j), t to tau[j].  Returns the number of steps.
template <bool kPivot>
__device__ int factor(cg::cluster_group &cluster, Qr &q, int kmax, double tol2, double2 *QV, double2 *tau) {
  __shared__ double red[kQW];
  __shared__ double2 s_t;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int M = q.M, N = q.N, C = q.C, rank = q.rank;
  for (int j = 0; j < kmax; ++j) {
    const volatile double *vn1 = q.n1[j & 1];
    // pivot: first column of largest remaining norm, by every warp
    int pc = j, bp = j;
    if (kPivot) {
      long long best = -1;
      bp = N;
      for (int p = j + lane; p < N; p += 32) {
        const long long b = __double_as_longlong(vn1[q.perm[p]]);
        if (b > best) {
          best = b;
          bp = p;
        }
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        const long long ob = __shfl_xor_sync(0xffffffffu, best, o);
        const int op = __shfl_xor_sync(0xffffffffu, bp, o);
        if (ob > best || (ob == best && op < bp)) {
          best = ob;
          bp = op;
        }
      }
      if (!(best >= 0 && __longlong_as_double(best) > tol2)) return j;  // uniform over the cluster
      pc = q.perm[bp];
    }
    // the column, as the reflector's tail, and its squared norm below row j
    const double2 *src = q.own ? cluster.map_shared_rank(q.own, pc % C) + (size_t)(pc / C) * M : q.glob + (size_t)M * pc;
    double acc = 0.0;
    for (int r = j + tid; r < M; r += kQThreads) {
      const double2 x = q.own ? src[r] : __ldcg(src + r);
      q.v[r] = x;
      if (r > j) {
        acc = fma(x.x, x.x, fma(x.y, x.y, acc));
        if (rank == 0) QV[r + (size_t)M * j] = x;
      }
    }
    if (warp * 32 < M - j) acc = wsum(acc);
    if (lane == 0) red[warp] = acc;
    __syncthreads();
    if (warp == 0) {
      const int parts = min(kQW, (M - j + 31) / 32);
      double xn = 0.0;
      for (int w = 0; w < parts; ++w) xn += red[w];
      const double2 a = q.v[j];
      double2 t = make_double2(0.0, 0.0), s = make_double2(1.0, 0.0);
      double beta = a.x;
      if (!(xn == 0.0 && a.y == 0.0)) {
        beta = -copysign(sqrt(fma(a.x, a.x, fma(a.y, a.y, xn))), a.x);
        s = make_double2(a.x - beta, a.y);
        const double f = -1.0 / (beta * fma(s.x, s.x, s.y * s.y));
        t = make_double2(f * s.x, -f * s.y);
      }
      if (lane == 0) {
        s_t = t;
        q.v[j] = s;
        q.beta[j] = beta;
        if (kPivot) {
          const int a0 = q.perm[j];
          q.perm[j] = pc;
          q.perm[bp] = a0;
          q.pos[pc] = j;
          if (bp != j) q.pos[a0] = bp;
        }
        if (rank == 0) {
          QV[j + (size_t)M * j] = s;
          tau[j] = t;
        }
      }
    }
    __syncthreads();
    // H^H on the remaining own columns, a warp each
    const double2 t = s_t;
    for (int c = rank + C * warp; c < N; c += C * kQW) {
      if ((kPivot ? q.pos[c] : c) <= j) continue;
      double2 *x = q.column(c);
      double wr = 0.0, wi = 0.0;  // v^H x
      for (int r = j + lane; r < M; r += 32) {
        const double2 a = x[r], v = q.v[r];
        wr = fma(v.x, a.x, fma(v.y, a.y, wr));
        wi = fma(v.x, a.y, fma(-v.y, a.x, wi));
      }
      wsum2(wr, wi, lane);
      const double fr = fma(t.x, wr, -t.y * wi), fi = fma(t.x, wi, t.y * wr);
      double2 top = make_double2(0.0, 0.0);
      for (int r = j + lane; r < M; r += 32) {
        const double2 v = q.v[r];
        double2 a = x[r];
        a.x = fma(-v.x, fr, fma(v.y, fi, a.x));
        a.y = fma(-v.x, fi, fma(-v.y, fr, a.y));
        x[r] = a;
        if (r == j) top = a;
      }
      if (kPivot) {  // ZLAQP2's norm downdate, on squares
        double left = 0.0;
        bool again = false;
        if (lane == 0) {
          const double was = vn1[c];
          left = fma(-top.x, top.x, fma(-top.y, top.y, was));
          again = was != 0.0 && !(left > 1.4901161193847656e-08 * q.n2[c]);
          if (was == 0.0) left = 0.0;
        }
        if (__shfl_sync(0xffffffffu, (int)again, 0)) {
          left = 0.0;
          for (int r = j + 1 + lane; r < M; r += 32) left = fma(x[r].x, x[r].x, fma(x[r].y, x[r].y, left));
          left = wsum(left);
          if (lane == 0) q.n2[c] = left;
        }
        left = __shfl_sync(0xffffffffu, left, 0);
        if (lane < C) *q.of(cluster, q.n1[(j + 1) & 1] + c, lane) = left;
      }
    }
    if (C > 1)
      cluster.sync();
    else
      __syncthreads();
  }
  return kmax;
}
}  // namespace

// ---------------------------------------------------------------------------
// 1., 2. both QRs: Q's reflectors to S.V (ld m), Q2's to aux + n^2 (ld n), X = R2^H to S.X
// (ld m, rows below k), Z = I to aux + 2 n^2 (ld n), and the Jacobi problem
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kQThreads, 1) k_qrj_factor(Slot *slots, JacobiProblem<double> *jp, const double *nrm,
                                                             const int *path, int in_smem, int scr_smem) {
  cg::cluster_group cluster = cg::this_cluster();
  const int s = blockIdx.y, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (path[s] != kPathQRJ) {  // the bidiagonal route: no Jacobi problem for this slot
    if (blockIdx.x == 0 && tid == 0) jp[s].n = 0;
    return;  // uniform per cluster
  }
  // the others' shared memory may be accessed once they are known to run: the norms below
  // are stored to every CTA
  cluster.sync();
  const Slot S = slots[s];
  const int m = S.cp->m, n = S.cp->n, mx = max(m, n);
  extern __shared__ __align__(16) char sh[];
  Qr q;
  q.C = (int)cluster.num_blocks();
  q.rank = (int)cluster.block_rank();
  double2 *A = S.aux, *QV2 = S.aux + (size_t)n * n, *Z = S.aux + 2 * (size_t)n * n;
  q.stride = qr_scratch(mx);
  q.scr = scr_smem ? nullptr : reinterpret_cast<char *>(Z);  // C stride <= 3 n^2 doubles: n > 4000 here
  q.place(scr_smem ? sh : q.scr + q.rank * q.stride, mx);
  q.own = in_smem ? reinterpret_cast<double2 *>(sh + qr_scratch(mx)) : nullptr;
  q.M = m;
  q.N = n;
  q.glob = S.X;
  // scaled to norm 1 by a power of two, so that no square leaves the range
  const double norm = nrm[s];
  const int e = norm > 0.0 && norm < INFINITY ? max(-1000, min(1000, ((__double2hiint(norm) >> 20) & 0x7ff) - 1023)) : 0;
  const double down = pow2(-e), up = pow2(e);
  for (int c = q.rank + q.C * warp; c < n; c += q.C * kQW) {
    double2 *x = q.column(c);
    double acc = 0.0;
    for (int r = lane; r < m; r += 32) {
      double2 a = S.X[r + (size_t)m * c];
      a = make_double2(a.x * down, a.y * down);
      x[r] = a;
      acc = fma(a.x, a.x, fma(a.y, a.y, acc));
    }
    acc = wsum(acc);
    if (lane == 0) q.n2[c] = acc;
    if (lane < q.C) *q.of(cluster, q.n1[0] + c, lane) = acc;
  }
  for (int c = tid; c < n; c += kQThreads) q.perm[c] = q.pos[c] = c;
  cluster.sync();
  const double tol = kNegligibleColumn * (norm * down);
  const int k = factor<true>(cluster, q, min(m, n), tol * tol, S.V, S.tau);
  // A = R^H (n x k, ld n)
  for (int c = q.rank + q.C * warp; c < n; c += q.C * kQW) {
    const int p = q.pos[c];
    const double2 *x = q.column(c);
    for (int r = lane; r < k; r += 32) {
      double2 a = make_double2(0.0, 0.0);
      if (r < p) a = make_double2(x[r].x, -x[r].y);
      if (r == p) a = make_double2(q.beta[p], 0.0);
      A[p + (size_t)n * r] = a;
    }
    if (lane == 0) S.jpvt[p] = c;
  }
  if (q.rank == 0 && tid == 0) {
    S.cp->k = k;
    JacobiProblem<double> P;
    P.X = S.X;
    P.V = Z;
    P.m = k;
    P.n = k;
    P.ldx = m > 0 ? m : 1;
    P.ldv = n > 0 ? n : 1;
    const double f = kNegligibleColumn * norm;
    P.floor = f * f;
    jp[s] = P;
  }
  cluster.sync();
  q.M = n;
  q.N = k;
  q.glob = A;
  if (q.own)
    for (int c = q.rank + q.C * warp; c < k; c += q.C * kQW)
      for (int r = lane; r < n; r += 32) q.column(c)[r] = __ldcg(A + r + (size_t)n * c);
  cluster.sync();
  factor<false>(cluster, q, k, 0.0, QV2, S.taup);
  // X = R2^H by rows: row c of X is column c of R2, conjugated
  for (int c = q.rank + q.C * warp; c < k; c += q.C * kQW) {
    const double2 *x = q.column(c);
    for (int r = lane; r < k; r += 32) {
      double2 a = make_double2(0.0, 0.0);
      if (r < c) a = make_double2(x[r].x * up, -x[r].y * up);
      if (r == c) a = make_double2(q.beta[c] * up, 0.0);
      S.X[c + (size_t)m * r] = a;
    }
  }
  cluster.sync();  // the scratch may lie in Z
  for (int c = q.rank + q.C * warp; c < k; c += q.C * kQW)
    for (int r = lane; r < k; r += 32) Z[r + (size_t)n * c] = make_double2(r == c ? 1.0 : 0.0, 0.0);
}

// ---------------------------------------------------------------------------
// 4. S.X(:, i) = Q [W(:, i) sigma_i; 0] (z = 0) and Y(:, i) = Q2 [Z(:, i); 0] (z = 1), in
// place, one warp per column; sigma_i = |X(:, i)|
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) k_qrj_apply_q(Slot *slots, const int *path, int in_smem) {
  const int s = blockIdx.y;
  if (path[s] != kPathQRJ) return;
  const Slot S = slots[s];
  const int n = S.cp->n, k = S.cp->k, left = blockIdx.z == 0;
  const int rows = left ? S.cp->m : n;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int i = blockIdx.x * (blockDim.x >> 5) + warp;
  if (i >= k) return;
  double2 *mat = (left ? S.X : S.aux + 2 * (size_t)n * n) + (size_t)rows * i;
  const double2 *QV = left ? S.V : S.aux + (size_t)n * n, *tau = left ? S.tau : S.taup;
  extern __shared__ double2 ys[];
  double2 *y = in_smem ? ys + (size_t)rows * warp : mat;
  double acc = 0.0;
  for (int r = lane; r < rows; r += 32) {
    const double2 v = r < k ? mat[r] : make_double2(0.0, 0.0);
    acc = fma(v.x, v.x, fma(v.y, v.y, acc));
    y[r] = v;
  }
  if (left) {
    acc = sqrt(wsum(acc));
    if (lane == 0) S.vn[i] = acc;
  }
  __syncwarp();
  for (int j = k - 1; j >= 0; --j) {  // Q y = H_0 (H_1 (... H_{k-1} y)), H = I - conj(t) v v^H
    const double2 *vj = QV + (size_t)rows * j;
    const double2 t = tau[j];
    double wr = 0.0, wi = 0.0;
    for (int r = j + lane; r < rows; r += 32) {
      const double2 a = y[r], v = vj[r];
      wr = fma(v.x, a.x, fma(v.y, a.y, wr));
      wi = fma(v.x, a.y, fma(-v.y, a.x, wi));
    }
    wsum2(wr, wi, lane);
    const double fr = fma(t.x, wr, t.y * wi), fi = fma(t.x, wi, -t.y * wr);
    for (int r = j + lane; r < rows; r += 32) {
      const double2 v = vj[r];
      double2 a = y[r];
      a.x = fma(-v.x, fr, fma(v.y, fi, a.x));
      a.y = fma(-v.x, fi, fma(-v.y, fr, a.y));
      y[r] = a;
    }
    __syncwarp();
  }
  if (in_smem)
    for (int r = lane; r < rows; r += 32) mat[r] = y[r];
}

// V(jpvt(c), i) = Y(c, i); zero where sigma_i is
__global__ void k_qrj_store(Slot *slots, const int *path) {
  const int s = blockIdx.y;
  if (path[s] != kPathQRJ) return;
  const Slot S = slots[s];
  const int n = S.cp->n, k = S.cp->k;
  const double2 *Y = S.aux + 2 * (size_t)n * n;
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < (size_t)n * k; e += (size_t)gridDim.x * blockDim.x) {
    const int c = (int)(e % n), i = (int)(e / n);
    S.V[(size_t)S.jpvt[c] + (size_t)n * i] = S.vn[i] > 0.0 ? Y[e] : make_double2(0.0, 0.0);
  }
}

// ---------------------------------------------------------------------------
// host orchestration (dense batch, after launch_dense_prepare)
// ---------------------------------------------------------------------------
int run_qrj(tebd_handle *h, int nb) {
  cudaStream_t st = h->stream;
  int rc, mx = 1, kx = 1, nqr = 0;
  size_t nk = 1;
  for (int s = 0; s < nb; ++s) {
    if (h->path_h[s] != kPathQRJ) continue;
    const Compact &c = h->cps[s];
    ++nqr;
    mx = std::max(mx, std::max(c.m, c.n));
    kx = std::max(kx, std::min(c.m, c.n));
    nk = std::max(nk, (size_t)c.n * std::min(c.m, c.n));
  }
  JacobiProblem<double> *jp = reinterpret_cast<JacobiProblem<double> *>(h->jprob_d);
  // 1., 2. the two QRs: as many CTAs per bond as the GPU has for the batch, with at least 16
  // columns each; more where the columns need the shared memory
  {
    int C = std::max(1, std::min(std::min(152 / nqr, (mx + 15) / 16), kMaxC));
    while (C < kMaxC && qr_scratch(mx) + qr_columns(mx, C) > kSmemMax) ++C;
    const int scr_smem = qr_scratch(mx) <= kSmemMax, in_smem = qr_scratch(mx) + qr_columns(mx, C) <= kSmemMax;
    if ((rc = check_cuda(h, cudaFuncSetAttribute(k_qrj_factor, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemMax),
                         "QR shared memory")))
      return rc;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(C, nb, 1);
    cfg.blockDim = dim3(kQThreads, 1, 1);
    cfg.dynamicSmemBytes = (scr_smem ? qr_scratch(mx) : 0) + (in_smem ? qr_columns(mx, C) : 0);
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = C;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (h->profiling) cudaEventRecord(h->ev[0], st);
    rc = check_cuda(h, cudaLaunchKernelEx(&cfg, k_qrj_factor, h->slots_d, jp, (const double *)h->nrm,
                                          (const int *)h->path_d, in_smem, scr_smem), "QR launch");
    if (rc) return rc;
    TEBD_LAUNCHED(h);
    if (h->profiling) {
      cudaEventRecord(h->ev[1], st);
      if ((rc = check_cuda(h, cudaStreamSynchronize(st), "QR"))) return rc;
      float ms = 0.f;
      if (cudaEventElapsedTime(&ms, h->ev[0], h->ev[1]) == cudaSuccess) h->stats.qr_ms += ms;
    }
  }
  // 3. Jacobi on R2^H; the default tolerance follows each problem's rank
  const int cap = h->opts.max_sweeps > 0 ? h->opts.max_sweeps : 60;
  if ((rc = jacobi_persistent_double(h, jp, nb, kx, h->opts.jacobi_tol > 0 ? h->opts.jacobi_tol : 0.0, cap))) return rc;
  // 4. U and V
  int warps = 8;
  while (warps > 1 && 16 * (size_t)mx * warps > kSmemMax) warps /= 2;
  const size_t smem = 16 * (size_t)mx * warps <= kSmemMax ? 16 * (size_t)mx * warps : 0;
  if ((rc = check_cuda(h, cudaFuncSetAttribute(k_qrj_apply_q, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemMax),
                       "back-transformation shared memory")))
    return rc;
  k_qrj_apply_q<<<dim3((kx + warps - 1) / warps, nb, 2), 32 * warps, smem, st>>>(h->slots_d, h->path_d, smem > 0);
  TEBD_LAUNCHED(h);
  k_qrj_store<<<dim3((unsigned)std::min<size_t>((nk + 255) / 256, 512), nb), 256, 0, st>>>(h->slots_d, h->path_d);
  TEBD_LAUNCHED(h);
  return check_cuda(h, cudaGetLastError(), "QRJ launch");
}

// ranks and flops of a finished batch's bonds on this route
void qrj_count(tebd_handle *h, int nb, const Compact *cp) {
  for (int s = 0; s < nb; ++s) {
    if (h->path_h[s] != kPathQRJ) continue;
    const double m = cp[s].m, n = cp[s].n, k = cp[s].k;
    // 16 flop per element of each reflector application: w = v^H x and x -= f v
    auto qr = [](double M, double N, double K) {
      return 16.0 * (K * M * N - (M + N) * K * (K - 1) / 2.0 + K * (K - 1) * (2 * K - 1) / 6.0);
    };
    h->stats.qr_flops += qr(m, n, k) + qr(n, k, k);
    h->stats.qr_flops += 16.0 * (m + n) * k * k;  // U = Q [W; 0], V = Q2 [Z; 0] (upper bound)
    h->stats.rank_sum += cp[s].k;
  }
}

}  // namespace tebd
