// obs.cu -- observables of the device-resident chain (the reference's
// VidalCore_v_2.0/observables_module.f90), so that a host does not download the
// chain to measure it:
//   tebd_single_site_rho   SingleSiteDensityMatrix / FormSingleSiteRho      :95-131
//   tebd_one_site_expval   OneSiteExpVal_c (complex Op), _r (real Op)        :194-252
//   tebd_two_site_rho      ThetaKernal + TwoSiteRho on sites link, link+1   :704-832
//   tebd_local_energy      LocalEnergy (open boundary)                       :1346-1387
//   tebd_total_energy      TotalEnergy (open boundary)                       :1432-1466
//   tebd_inner_product     InnerProduct                                     :1031-1089
//   tebd_chain_entropy     ChainEntropy for every link                       :1583-1602
// Sums run in a fixed order (deterministic), not in the reference's loop order,
// so results agree with it to rounding.  Two-site density matrices reuse the
// update's batched Theta formation (k_compact + k_theta_form, no gate)
// on the handle's SVD slots, so observables and updates of one handle are
// serialised on its stream.
#include <math.h>
#include <string.h>

#include <algorithm>
#include <string>
#include <vector>

#include "tebd_internal.cuh"

namespace tebd {

namespace {

constexpr int kObsThreads = 256;

inline unsigned cdiv(size_t a, size_t b) { return (unsigned)((a + b - 1) / b); }

__device__ __forceinline__ void cacc(double2 &acc, double2 x, double2 y, double w) {  // acc += w x conj(y)
  const double re = x.x * y.x + x.y * y.y, im = x.y * y.x - x.x * y.y;
  acc.x = fma(w, re, acc.x);
  acc.y = fma(w, im, acc.y);
}

// rho_s(i,j) = sum_{a,b} l0(a)^2 l1(b)^2 G(a,i,b) conj(G(a,j,b)), i <= j (the rest is its
// conjugate).  A CTA takes a part of the columns b of one site, its threads the rows a
// (neighbouring in memory), every G entry read once; the CTA's sums go to part[site][CTA],
// added in that order by k_obs_rho1_sum.  One CTA per site with the d^2 entries split
// over its threads was bound by the latency of its reads (chi = 512: 24 ms for 16 sites;
// now 0.86 ms; chi = 128, 64 sites: 1.56 -> 0.34 ms).
template <int kD>
__global__ void __launch_bounds__(kObsThreads) k_obs_rho1(const double2 *gam, const double *lam, double2 *part,
                                                          int chi, int cols) {
  constexpr int kPairs = kD * (kD + 1) / 2;
  const int s = blockIdx.x, b0 = blockIdx.y * cols, b1 = min(chi, b0 + cols);
  const double2 *G = gam + (size_t)s * chi * kD * chi;
  const double *l0 = lam + (size_t)s * chi, *l1 = lam + (size_t)(s + 1) * chi;
  double2 acc[kPairs];
#pragma unroll
  for (int q = 0; q < kPairs; ++q) acc[q] = make_double2(0.0, 0.0);
  for (size_t e = threadIdx.x; e < (size_t)chi * (b1 - b0); e += kObsThreads) {
    const int a = (int)(e % chi), b = b0 + (int)(e / chi);
    const double w = l0[a] * l0[a] * l1[b] * l1[b];
    if (w == 0.0) continue;
    double2 g[kD];
#pragma unroll
    for (int i = 0; i < kD; ++i) g[i] = G[a + (size_t)chi * (i + (size_t)kD * b)];
    int q = 0;
#pragma unroll
    for (int i = 0; i < kD; ++i)
#pragma unroll
      for (int j = i; j < kD; ++j) cacc(acc[q++], g[i], g[j], w);
  }
  __shared__ double2 red[kObsThreads / 32][kPairs];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
  for (int q = 0; q < kPairs; ++q) {
    double2 v = acc[q];
    for (int o = 16; o > 0; o >>= 1) {
      v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
      v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
    }
    if (lane == 0) red[warp][q] = v;
  }
  __syncthreads();
  if (threadIdx.x < kPairs) {
    double2 v = make_double2(0.0, 0.0);
    for (int w = 0; w < kObsThreads / 32; ++w) {
      v.x += red[w][threadIdx.x].x;
      v.y += red[w][threadIdx.x].y;
    }
    part[((size_t)s * gridDim.y + blockIdx.y) * kPairs + threadIdx.x] = v;
  }
}

__global__ void k_obs_rho1_sum(const double2 *part, double2 *rho, int d, int nparts) {
  const int s = blockIdx.x, t = threadIdx.x, pairs = d * (d + 1) / 2;
  if (t >= d * d) return;
  const int i = min(t % d, t / d), j = max(t % d, t / d);
  const int q = i * d - i * (i - 1) / 2 + (j - i);
  double2 v = make_double2(0.0, 0.0);
  for (int c = 0; c < nparts; ++c) {
    const double2 p = part[((size_t)s * nparts + c) * pairs + q];
    v.x += p.x;
    v.y += p.y;
  }
  if (t % d > t / d) v.y = -v.y;  // rho(i,j), i > j: the conjugate of rho(j,i)
  rho[(size_t)s * d * d + t] = v;
}

// rho2[(i,j),(l,k)] = sum_{a,b} Theta(a,i,j,b) conj(Theta(a,l,k,b)) from the slot's
// compacted Theta X (row i*r0 + a', column j*r2 + b', ld m = d*r0); row index
// i*d + j, column l*d + k (the gate's order), column-major d^2 x d^2.  A CTA takes a
// part of the (a', b') pairs of one bond, staged kRhoE at a time with their d^2 entries,
// its threads the (row, column) pairs with row <= column; sums to part[bond][CTA], added
// in order by k_obs_rho2_sum.  (One CTA per row, two global reads per multiply-add,
// took 4.2 ms for 32 bonds of 640 x 640; now 3.1 ms, nearly the FP64 pipe's 2.6.)
constexpr int kRhoE = 16;
__global__ void __launch_bounds__(kObsThreads) k_obs_rho2(const Slot *slots, double2 *part, int d) {
  extern __shared__ double2 th[];  // kRhoE x d^2
  const int s = blockIdx.y;
  const Slot S = slots[s];
  const Compact cp = *S.cp;
  const int r0 = cp.r0, r2 = cp.r2, m = cp.m, d2 = d * d, pairs = d2 * (d2 + 1) / 2;
  const int total = r0 * r2, per = (total + gridDim.x - 1) / gridDim.x;
  const int e0 = blockIdx.x * per, e1 = min(total, e0 + per);
  double2 *out = part + ((size_t)s * gridDim.x + blockIdx.x) * pairs;
  // pairs of one pass: as many as the threads hold accumulators for, two each
  for (int p0 = 0; p0 < pairs; p0 += 2 * kObsThreads) {
    int row[2], col[2];
    double2 acc[2] = {make_double2(0.0, 0.0), make_double2(0.0, 0.0)};
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      int q = p0 + u * kObsThreads + threadIdx.x, r = 0;
      if (q >= pairs) q = pairs - 1;
      while (q >= d2 - r) {
        q -= d2 - r;
        ++r;
      }
      row[u] = r;
      col[u] = r + q;
    }
    // of a warp: whether it has pairs at all (small d leaves most without, and the FP64 pipe free)
    const int w0 = p0 + (threadIdx.x & ~31);
    const bool one = w0 < pairs, two = w0 + kObsThreads < pairs;
    for (int e = e0; e < e1; e += kRhoE) {
      const int ne = min(kRhoE, e1 - e);
      __syncthreads();
      for (int t = threadIdx.x; t < kRhoE * d2; t += kObsThreads) {
        const int x = t % kRhoE, ij = t / kRhoE;
        double2 v = make_double2(0.0, 0.0);
        if (x < ne) {
          const int a = (e + x) % r0, b = (e + x) / r0;
          v = S.X[((ij / d) * r0 + a) + (size_t)m * ((ij % d) * r2 + b)];
        }
        th[x * d2 + ij] = v;
      }
      __syncthreads();
      for (int x = 0; x < ne; ++x) {
        if (one) cacc(acc[0], th[x * d2 + row[0]], th[x * d2 + col[0]], 1.0);
        if (two) cacc(acc[1], th[x * d2 + row[1]], th[x * d2 + col[1]], 1.0);
      }
    }
#pragma unroll
    for (int u = 0; u < 2; ++u)
      if (p0 + u * kObsThreads + threadIdx.x < pairs) out[p0 + u * kObsThreads + threadIdx.x] = acc[u];
  }
}

__global__ void __launch_bounds__(kObsThreads) k_obs_rho2_sum(const Slot *slots, const double2 *part, double2 *rho2,
                                                              int d, int nparts) {
  const int s = blockIdx.y, d2 = d * d, pairs = d2 * (d2 + 1) / 2;
  const int t = blockIdx.x * kObsThreads + threadIdx.x;
  if (t >= d2 * d2) return;
  const int row = t % d2, col = t / d2, r = min(row, col), c = max(row, col);
  const int q = r * d2 - r * (r - 1) / 2 + (c - r);
  double2 v = make_double2(0.0, 0.0);
  for (int k = 0; k < nparts; ++k) {
    const double2 p = part[((size_t)s * nparts + k) * pairs + q];
    v.x += p.x;
    v.y += p.y;
  }
  if (row > col) v.y = -v.y;
  if (slots[s].cp->bad) v = make_double2(nan(""), nan(""));
  rho2[(size_t)s * d2 * d2 + t] = v;
}

// S(link) = -sum_{lambda != 0} lambda^2 ln|lambda^2| / ln(d), one warp per link
__global__ void k_obs_entropy(const double *lam, double *ent, int chi, int nlinks, double inv_logd) {
  const int link = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (link >= nlinks) return;
  const double *l = lam + (size_t)link * chi;
  double a = 0.0;
  for (int k = lane; k < chi; k += 32) {
    const double v = l[k];
    if (v != 0.0) a -= v * v * log(fabs(v * v));
  }
  for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
  if (lane == 0) ent[link] = a * inv_logd;
}

// One product of the overlap's chains: C(m, n) at C[m + ldc n] = sum_k A(m, k) B(k, n),
// A(m, k) = a[m am + k ak] (conjugated if conj_a) times sa[(m or k) / div], B(k, n) =
// b[k bk + n bn] times sb[(k or n) / div] where these are given, in FP64.
struct ObsGemm {
  int M, N, K, am, ak, bk, bn, ldc;
  const double2 *a, *b;
  double2 *c;
  bool conj_a, sa_k, sb_k;  // scale index: k, else m (n)
  const double *sa, *sb;
  int sa_div, sb_div;
};
struct ObsGemms {
  ObsGemm g[2];
};
// 16 x 16 tiles: the products are as small as chi x chi x (d chi), and a site's two
// products wait for the previous site's, so a chain needs every SM on one product
// (64 x 64 tiles left 4 CTAs on the second product: 3.2 ms per site at d = 5, chi = 128,
// 204 ms for 64 sites; now 19 ms, 10 of them the FP64 pipe's).
constexpr int kGT = 16, kGK = 16, kGThreads = 64;
__global__ void __launch_bounds__(kGThreads) k_obs_gemm(const ObsGemms both) {
  __shared__ double2 As[kGK][kGT + 1], Bs[kGK][kGT + 1];
  const ObsGemm &p = both.g[blockIdx.z];
  const int m0 = blockIdx.x * kGT, n0 = blockIdx.y * kGT;
  if (m0 >= p.M || n0 >= p.N) return;  // uniform
  const int t = threadIdx.x, tx = t & 7, ty = t >> 3;  // rows ty + 8 u, columns tx + 8 v
  double2 acc[2][2];
#pragma unroll
  for (int u = 0; u < 2; ++u)
#pragma unroll
    for (int v = 0; v < 2; ++v) acc[u][v] = make_double2(0.0, 0.0);
  for (int k0 = 0; k0 < p.K; k0 += kGK) {
    __syncthreads();
    for (int e = t; e < kGK * kGT; e += kGThreads) {
      int x = e % kGT, k = e / kGT;  // the index that is contiguous in memory runs fastest
      if (p.ak == 1) {
        k = e % kGK;
        x = e / kGK;
      }
      double2 v = make_double2(0.0, 0.0);
      if (m0 + x < p.M && k0 + k < p.K) {
        v = p.a[(size_t)(m0 + x) * p.am + (size_t)(k0 + k) * p.ak];
        if (p.sa) {
          const double w = p.sa[(p.sa_k ? k0 + k : m0 + x) / p.sa_div];
          v = make_double2(v.x * w, v.y * w);
        }
        if (p.conj_a) v.y = -v.y;
      }
      As[k][x] = v;
      x = e % kGT;
      k = e / kGT;
      if (p.bk == 1) {
        k = e % kGK;
        x = e / kGK;
      }
      v = make_double2(0.0, 0.0);
      if (n0 + x < p.N && k0 + k < p.K) {
        v = p.b[(size_t)(k0 + k) * p.bk + (size_t)(n0 + x) * p.bn];
        if (p.sb) {
          const double w = p.sb[(p.sb_k ? k0 + k : n0 + x) / p.sb_div];
          v = make_double2(v.x * w, v.y * w);
        }
      }
      Bs[k][x] = v;
    }
    __syncthreads();
#pragma unroll 4
    for (int kk = 0; kk < kGK; ++kk) {
      double2 av[2], bv[2];
#pragma unroll
      for (int u = 0; u < 2; ++u) av[u] = As[kk][ty + 8 * u];
#pragma unroll
      for (int v = 0; v < 2; ++v) bv[v] = Bs[kk][tx + 8 * v];
#pragma unroll
      for (int u = 0; u < 2; ++u)
#pragma unroll
        for (int v = 0; v < 2; ++v) {
          acc[u][v].x = fma(av[u].x, bv[v].x, fma(-av[u].y, bv[v].y, acc[u][v].x));
          acc[u][v].y = fma(av[u].x, bv[v].y, fma(av[u].y, bv[v].x, acc[u][v].y));
        }
    }
  }
#pragma unroll
  for (int u = 0; u < 2; ++u)
#pragma unroll
    for (int v = 0; v < 2; ++v) {
      const int m = m0 + ty + 8 * u, n = n0 + tx + 8 * v;
      if (m < p.M && n < p.N) p.c[m + (size_t)p.ldc * n] = acc[u][v];
    }
}

// sum over all entries of E F (one CTA, fixed order)
__global__ void __launch_bounds__(kObsThreads) k_obs_close(const double2 *E, const double2 *F, size_t n, double2 *out) {
  __shared__ double2 part[kObsThreads];
  double2 acc = make_double2(0.0, 0.0);
  for (size_t e = threadIdx.x; e < n; e += kObsThreads) {
    const double2 x = E[e], y = F[e];
    acc.x = fma(x.x, y.x, fma(-x.y, y.y, acc.x));
    acc.y = fma(x.x, y.y, fma(x.y, y.x, acc.y));
  }
  part[threadIdx.x] = acc;
  __syncthreads();
  for (int o = kObsThreads / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) {
      part[threadIdx.x].x += part[threadIdx.x + o].x;
      part[threadIdx.x].y += part[threadIdx.x + o].y;
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) *out = part[0];
}

__global__ void k_obs_unit(double2 *E, int chi, double *e1) {  // E = e1 e1^T, e1 = unit vector
  for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < (size_t)chi * chi;
       q += (size_t)gridDim.x * blockDim.x)
    E[q] = make_double2(q == 0 ? 1.0 : 0.0, 0.0);
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < chi; q += gridDim.x * blockDim.x)
    e1[q] = q == 0 ? 1.0 : 0.0;
}

}  // namespace

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
// Workspace: rho1 (L d^2) or rho2 (nslots d^4) results with the CTAs' partial sums, or,
// for each of the two chains of an overlap, transfer matrices E, E' (chi^2 each) and T
// (chi x d chi) with a unit vector (chi doubles), or the entropies (L+1).
constexpr int kRho1Parts = 32;  // CTAs per site, per bond
constexpr int kRho2Parts = 10;  // of a batch of 16 bonds or more; fewer bonds share out kRho2All
constexpr int kRho2All = 152;
static size_t rho2_parts(const tebd_handle *h) { return std::max(kRho2Parts * h->nslots, kRho2All); }
static int obs_ws(tebd_handle *h, size_t bytes) {
  if (h->obs_bytes >= bytes) return TEBD_OK;
  cudaFree(h->obs_buf);
  h->obs_buf = nullptr;
  h->obs_bytes = 0;
  int rc = check_cuda(h, cudaMalloc(&h->obs_buf, bytes), "alloc observables workspace");
  if (rc == TEBD_OK) h->obs_bytes = bytes;
  return rc;
}

static int obs_begin(tebd_handle *h) {
  int rc = check_cuda(h, cudaSetDevice(h->device), "cudaSetDevice");
  if (rc) return rc;
  const size_t n = (size_t)h->chi, d2 = (size_t)h->d * h->d;
  const size_t need = sizeof(double2) * std::max({(size_t)h->L * (d2 + kRho1Parts * d2),
                                                  (size_t)h->nslots * d2 * d2 + rho2_parts(h) * d2 * (d2 + 1) / 2,
                                                  2 * (2 * n * n + n * h->d * n) + 1}) +
                      sizeof(double) * (n + h->L + 1) + 1024;
  return obs_ws(h, need);
}

static int obs_finish(tebd_handle *h, const char *what) {
  int rc = check_cuda(h, cudaGetLastError(), what);
  if (rc) return rc;
  return check_cuda(h, cudaStreamSynchronize(h->stream), what);
}

// rho2 of every bond in `links` (d^4 complex each, in list order) into `out`
static int obs_rho2(tebd_handle *h, const std::vector<int> &links, std::vector<double2> &out) {
  const int d = h->d, d2 = d * d, d4 = d2 * d2;
  out.assign((size_t)links.size() * d4, make_double2(0.0, 0.0));
  double2 *rho2_d = reinterpret_cast<double2 *>(h->obs_buf);
  // same-parity bonds share no site: odd links, then even links, nslots at a time
  std::vector<int> order;
  for (int par = 1; par >= 0; --par)
    for (size_t q = 0; q < links.size(); ++q)
      if ((links[q] & 1) == par) order.push_back((int)q);
  for (size_t base = 0; base < order.size();) {
    const int par = links[order[base]] & 1;
    std::vector<int> idx;
    while (base < order.size() && (int)idx.size() < h->nslots && (links[order[base]] & 1) == par)
      idx.push_back(order[base++]);
    const int nb = (int)idx.size();
    std::vector<int> lk(nb);
    for (int s = 0; s < nb; ++s) lk[s] = links[idx[s]];
    int rc;
    if ((rc = check_cuda(h, cudaMemcpyAsync(h->links_d, lk.data(), sizeof(int) * nb, cudaMemcpyHostToDevice,
                                            h->stream),
                         "upload links")))
      return rc;
    if ((rc = check_cuda(h, cudaMemsetAsync(h->status_d, 0, sizeof(int) * 4, h->stream), "reset status")))
      return rc;
    if ((rc = launch_dense_prepare(h, nb, false))) return rc;
    double2 *part = rho2_d + (size_t)h->nslots * d4;
    // two CTAs per SM in a large batch, one in a small one (10 for a single bond of d = 3,
    // chi = 200 took 2.1 ms, 0.34 now); at least two stages of pairs each
    const int most = (int)cdiv((size_t)h->chi * h->chi, 2 * kRhoE);
    const int nparts = std::max(1, std::min(most, std::max(std::min(kRho2Parts, 304 / nb), kRho2All / nb)));
    k_obs_rho2<<<dim3(nparts, nb), kObsThreads, sizeof(double2) * kRhoE * d2, h->stream>>>(h->slots_d, part, d);
    TEBD_LAUNCHED(h);
    k_obs_rho2_sum<<<dim3(cdiv(d4, kObsThreads), nb), kObsThreads, 0, h->stream>>>(h->slots_d, part, rho2_d, d, nparts);
    TEBD_LAUNCHED(h);
    std::vector<double2> tmp((size_t)nb * d4);
    if ((rc = check_cuda(h, cudaMemcpyAsync(tmp.data(), rho2_d, sizeof(double2) * tmp.size(),
                                            cudaMemcpyDeviceToHost, h->stream),
                         "read two-site density matrices")))
      return rc;
    if ((rc = obs_finish(h, "two-site density matrices"))) return rc;
    if ((rc = tc_check(h))) return rc;
    for (int s = 0; s < nb; ++s)
      memcpy(out.data() + (size_t)idx[s] * d4, tmp.data() + (size_t)s * d4, sizeof(double2) * d4);
  }
  return TEBD_OK;
}

// Re Tr(H rho2) = Re sum_{a,b} H(a,b) rho2(b,a)  (TraceMatmul, TEBDtools_module.f90:401)
static double trace_matmul_re(const double *H, const double2 *rho2, int d2) {
  double acc = 0.0;
  for (int a = 0; a < d2; ++a)
    for (int b = 0; b < d2; ++b) {
      const double hr = H[2 * (a + (size_t)d2 * b)], hi = H[2 * (a + (size_t)d2 * b) + 1];
      const double2 r = rho2[b + (size_t)d2 * a];
      acc += hr * r.x - hi * r.y;
    }
  return acc;
}

}  // namespace tebd

using namespace tebd;

extern "C" int tebd_single_site_rho(tebd_handle *h, double *rho) {
  if (!h || !rho) return TEBD_ERR_ARG;
  int rc;
  if ((rc = obs_begin(h))) return rc;
  const size_t d2 = (size_t)h->d * h->d;
  double2 *rho_d = reinterpret_cast<double2 *>(h->obs_buf);
  double2 *part = rho_d + d2 * h->L;
  const int cols = (int)cdiv(h->chi, kRho1Parts), nparts = (int)cdiv(h->chi, cols);
  auto rho1 = [&](auto kern) { kern<<<dim3(h->L, nparts), kObsThreads, 0, h->stream>>>(h->gam, h->lam, part, h->chi, cols); };
  switch (h->d) {
    case 1: rho1(k_obs_rho1<1>); break;
    case 2: rho1(k_obs_rho1<2>); break;
    case 3: rho1(k_obs_rho1<3>); break;
    case 4: rho1(k_obs_rho1<4>); break;
    case 5: rho1(k_obs_rho1<5>); break;
    case 6: rho1(k_obs_rho1<6>); break;
    case 7: rho1(k_obs_rho1<7>); break;
    default: rho1(k_obs_rho1<8>); break;
  }
  TEBD_LAUNCHED(h);
  k_obs_rho1_sum<<<h->L, 64, 0, h->stream>>>(part, rho_d, h->d, nparts);
  TEBD_LAUNCHED(h);
  if ((rc = check_cuda(h, cudaMemcpyAsync(rho, rho_d, sizeof(double2) * d2 * h->L, cudaMemcpyDeviceToHost,
                                          h->stream),
                       "read single-site density matrices")))
    return rc;
  return obs_finish(h, "single-site density matrices");
}

static int one_site(tebd_handle *h, const double *op, bool real_op, double *out) {
  if (!h || !op || !out) return TEBD_ERR_ARG;
  const int d = h->d, d2 = d * d;
  std::vector<double2> rho((size_t)h->L * d2);
  int rc;
  if ((rc = tebd_single_site_rho(h, reinterpret_cast<double *>(rho.data())))) return rc;
  for (int s = 0; s < h->L; ++s) {  // Tr(Op rho) = sum_{i,j} Op(i,j) rho(j,i)
    double re = 0.0, im = 0.0;
    for (int i = 0; i < d; ++i)
      for (int j = 0; j < d; ++j) {
        const double2 r = rho[(size_t)s * d2 + j + (size_t)d * i];
        const double orr = real_op ? op[i + (size_t)d * j] : op[2 * (i + (size_t)d * j)];
        const double oi = real_op ? 0.0 : op[2 * (i + (size_t)d * j) + 1];
        re += orr * r.x - oi * r.y;
        im += orr * r.y + oi * r.x;
      }
    if (real_op) {
      out[s] = re;
    } else {
      out[2 * s] = re;
      out[2 * s + 1] = im;
    }
  }
  return TEBD_OK;
}

extern "C" int tebd_one_site_expval(tebd_handle *h, const double *op, double *exp_list) {
  return one_site(h, op, false, exp_list);
}

extern "C" int tebd_one_site_expval_r(tebd_handle *h, const double *op, double *exp_list) {
  return one_site(h, op, true, exp_list);
}

extern "C" int tebd_two_site_rho(tebd_handle *h, int link, double *rho2) {
  if (!h || !rho2) return TEBD_ERR_ARG;
  if (link < 1 || link > h->L - 1) return set_error(h, TEBD_ERR_ARG, "tebd_two_site_rho: link out of range");
  int rc;
  if ((rc = obs_begin(h))) return rc;
  std::vector<double2> out;
  const std::vector<int> one_link{link};
  if ((rc = obs_rho2(h, one_link, out))) return rc;
  memcpy(rho2, out.data(), sizeof(double2) * out.size());
  return TEBD_OK;
}

static int bond_energies(tebd_handle *h, int n_ops, const double *const *H, std::vector<double> &en) {
  if (!h || !H) return TEBD_ERR_ARG;
  if (n_ops < h->L - 1) return set_error(h, TEBD_ERR_ARG, "energy: need one bond operator per bond (L-1)");
  for (int l = 0; l < h->L - 1; ++l)
    if (!H[l]) return set_error(h, TEBD_ERR_ARG, "energy: null bond operator");
  int rc;
  if ((rc = obs_begin(h))) return rc;
  std::vector<int> links(h->L - 1);
  for (int l = 0; l < h->L - 1; ++l) links[l] = l + 1;
  std::vector<double2> rho2;
  if ((rc = obs_rho2(h, links, rho2))) return rc;
  const int d2 = h->d * h->d;
  en.resize(h->L - 1);
  for (int l = 0; l < h->L - 1; ++l) en[l] = trace_matmul_re(H[l], rho2.data() + (size_t)l * d2 * d2, d2);
  return TEBD_OK;
}

extern "C" int tebd_local_energy(tebd_handle *h, int n_ops, const double *const *H, double *energy) {
  if (!energy) return TEBD_ERR_ARG;
  std::vector<double> en;
  int rc = bond_energies(h, n_ops, H, en);
  if (rc) return rc;
  memcpy(energy, en.data(), sizeof(double) * en.size());
  return TEBD_OK;
}

extern "C" int tebd_total_energy(tebd_handle *h, int n_ops, const double *const *H, double *energy) {
  if (!energy) return TEBD_ERR_ARG;
  std::vector<double> en;
  int rc = bond_energies(h, n_ops, H, en);
  if (rc) return rc;
  double e = 0.0;
  for (double x : en) e += x;  // the reference's bond order
  *energy = e;
  return TEBD_OK;
}

extern "C" int tebd_inner_product(tebd_handle *left, tebd_handle *right, double *value) {
  if (!left || !right || !value) return TEBD_ERR_ARG;
  tebd_handle *h = left;
  if (left->L != right->L || left->d != right->d || left->chi != right->chi || left->device != right->device)
    return set_error(h, TEBD_ERR_ARG, "tebd_inner_product: chains differ in L, d, chi or device");
  int rc;
  if ((rc = obs_begin(h))) return rc;
  if (right != left && (rc = check_cuda(h, cudaStreamSynchronize(right->stream), "sync right chain"))) return rc;
  const int chi = h->chi, d = h->d, L = h->L;
  const size_t cc = (size_t)chi * chi, gsz = cc * d;
  double2 *ws = reinterpret_cast<double2 *>(h->obs_buf);
  // [0]: from the left, sites 1..half; [1]: from the right, sites L..half+1.  Both
  // chains take a site per step in the same launches; their products' ends meet in
  // sum_{x,y} E(x,y) F(x,y).
  double2 *E[2] = {ws, ws + cc}, *E2[2] = {ws + 2 * cc, ws + 3 * cc};
  double2 *T[2] = {ws + 4 * cc, ws + 4 * cc + gsz};
  double2 *res = ws + 4 * cc + 2 * gsz;
  double *e1 = reinterpret_cast<double *>(res + 1);
  cudaStream_t st = h->stream;
  for (int q = 0; q < 2; ++q) {
    k_obs_unit<<<64, 256, 0, st>>>(E[q], chi, e1);
    TEBD_LAUNCHED(h);
  }
  // the reference contracts the first site from left index 1 and the last site
  // into right index 1 (edge Lambdas e_1), without the edge Lambdas themselves
  auto lr = [&](int s) { return s == L - 1 ? e1 : right->lam + (size_t)(s + 1) * chi; };
  auto ll = [&](int s) { return s == L - 1 ? e1 : left->lam + (size_t)(s + 1) * chi; };
  const int half = (L + 1) / 2;
  for (int step = 0; step < half; ++step) {
    const int nz = L - 1 - step >= half ? 2 : 1, s0 = step, s1 = L - 1 - step;
    const double2 *gl0 = left->gam + s0 * gsz, *gr0 = right->gam + s0 * gsz;
    const double2 *gl1 = left->gam + s1 * gsz, *gr1 = right->gam + s1 * gsz;
    ObsGemms g = {};
    // T = E (Gamma_R Lambda_R): chi x (d chi), column i + d beta
    g.g[0] = {chi, d * chi, chi, 1, chi, 1, chi, chi, E[0], gr0, T[0], false, false, false, nullptr, lr(s0), 1, d};
    // T(alpha' + chi i, beta) = sum_beta' Gamma_R(alpha', i, beta') Lambda_R(beta') F(beta, beta')
    g.g[1] = {d * chi, chi, chi, 1, d * chi, chi, 1, d * chi, gr1, E[1], T[1], false, true, false, lr(s1), nullptr, 1, 1};
    k_obs_gemm<<<dim3(cdiv(nz == 2 ? (size_t)d * chi : chi, kGT), cdiv((size_t)d * chi, kGT), nz), kGThreads, 0, st>>>(g);
    TEBD_LAUNCHED(h);
    // E' = (Gamma_L Lambda_L)^H T over (gamma, i): chi x chi
    g.g[0] = {chi, chi, d * chi, d * chi, 1, 1, d * chi, chi, gl0, T[0], E2[0], true, false, false, ll(s0), nullptr, 1, 1};
    // F'(alpha, alpha') = sum_(i, beta) conj(Gamma_L(alpha, i, beta) Lambda_L(beta)) T(alpha', i, beta)
    g.g[1] = {chi, chi, d * chi, 1, chi, chi, 1, chi, gl1, T[1], E2[1], true, true, false, ll(s1), nullptr, d, 1};
    k_obs_gemm<<<dim3(cdiv(chi, kGT), cdiv(chi, kGT), nz), kGThreads, 0, st>>>(g);
    TEBD_LAUNCHED(h);
    for (int q = 0; q < nz; ++q) std::swap(E[q], E2[q]);
  }
  k_obs_close<<<1, kObsThreads, 0, st>>>(E[0], E[1], cc, res);
  TEBD_LAUNCHED(h);
  double2 v;
  if ((rc = check_cuda(h, cudaMemcpyAsync(&v, res, sizeof(double2), cudaMemcpyDeviceToHost, st), "read overlap")))
    return rc;
  if ((rc = obs_finish(h, "inner product"))) return rc;
  value[0] = v.x;
  value[1] = v.y;
  return TEBD_OK;
}

extern "C" int tebd_chain_entropy(tebd_handle *h, double *entropy) {
  if (!h || !entropy) return TEBD_ERR_ARG;
  int rc;
  if ((rc = obs_begin(h))) return rc;
  double *ent_d = reinterpret_cast<double *>(h->obs_buf);
  const int nl = h->L + 1;
  k_obs_entropy<<<cdiv(nl, 8), 256, 0, h->stream>>>(h->lam, ent_d, h->chi, nl, 1.0 / log((double)h->d));
  TEBD_LAUNCHED(h);
  if ((rc = check_cuda(h, cudaMemcpyAsync(entropy, ent_d, sizeof(double) * nl, cudaMemcpyDeviceToHost,
                                          h->stream),
                       "read entropies")))
    return rc;
  return obs_finish(h, "chain entropy");
}
