// theta_tc.cu -- FormTheta (VidalCore_v_2.0/local_operations_module.f90:184-211)
// as one batched complex product on the tensor cores.
//
// For every bond of the batch the two factors of Theta are gathered on the kept
// (compacted) indices into the slot's aux buffer, column-major and zero-filled to
// the batch's largest sizes:
//   A (m x r1): A[i*r0 + a', g'] = l0(a) G1(a, i, g),          a = idx0[a'], g = idx1[g']
//   B (r1 x n): B[g', j*r2 + b'] = l1(g) G2(g, j, b) l2(b),    b = idx2[b']
// and Theta = A B is written straight into the slot's X (m x n, ld m) -- the
// column order j*r2 + b' is the permuted order ReshapeTheta leaves, so nothing is
// moved afterwards.  The product runs in the handle's theta form: 3xTF32 (the
// split-precision form, ~FP32 accuracy) or S bf16 digit planes (S = 7: FP64
// class).  ThetaOperation, the norm and the SVD follow unchanged.
#include <stddef.h>

#include "tc_gemm.cuh"

namespace tebd {

constexpr double kThetaTcMin = 1 << 21;  // m n r1 from which Theta is formed on the tensor cores

int tc_reserve(tebd_handle *h, size_t bytes) {
  if (!h->tc_err) {
    int rc = check_cuda(h, cudaMalloc(&h->tc_err, sizeof(int)), "alloc tensor-core flag");
    if (rc) return rc;
    rc = check_cuda(h, cudaMemsetAsync(h->tc_err, 0, sizeof(int), h->stream), "clear tensor-core flag");
    if (rc) return rc;
  }
  if (bytes <= h->tc_ws_bytes) return TEBD_OK;
  int rc = check_cuda(h, cudaStreamSynchronize(h->stream), "tensor-core workspace");
  if (rc) return rc;
  cudaFree(h->tc_ws);
  h->tc_ws = nullptr;
  h->tc_ws_bytes = 0;
  rc = check_cuda(h, cudaMalloc(&h->tc_ws, bytes), "alloc tensor-core workspace");
  if (rc) return rc;
  h->tc_ws_bytes = bytes;
  return TEBD_OK;
}

void tc_events(tebd_handle *h, double flops, cudaEvent_t *e0, cudaEvent_t *e1) {
  *e0 = *e1 = nullptr;
  if (!h->profiling) return;
  const size_t need = 2 * (size_t)(h->tc_ev_used + 1);
  while (h->tc_ev.size() < need) {
    cudaEvent_t e;
    if (cudaEventCreate(&e) != cudaSuccess) {
      (void)cudaGetLastError();
      return;
    }
    h->tc_ev.push_back(e);
  }
  h->tc_ev_flops.resize(h->tc_ev.size() / 2);
  *e0 = h->tc_ev[2 * h->tc_ev_used];
  *e1 = h->tc_ev[2 * h->tc_ev_used + 1];
  h->tc_ev_flops[h->tc_ev_used] = flops;
  ++h->tc_ev_used;
}

void tc_collect(tebd_handle *h) {
  for (int i = 0; i < h->tc_ev_used; ++i) {
    float ms = 0.f;
    if (cudaEventElapsedTime(&ms, h->tc_ev[2 * i], h->tc_ev[2 * i + 1]) == cudaSuccess) {
      h->stats.tc_ms += ms;
      h->stats.tc_launches++;
      h->stats.tc_mma_flops += h->tc_ev_flops[i];
    }
  }
  (void)cudaGetLastError();
  h->tc_ev_used = 0;
}

void tc_free(tebd_handle *h) {
  for (cudaEvent_t e : h->tc_ev) cudaEventDestroy(e);
  h->tc_ev.clear();
  h->tc_ev_used = 0;
  cudaFree(h->tc_ws);
  cudaFree(h->tc_err);
  h->tc_ws = nullptr;
  h->tc_err = nullptr;
  h->tc_ws_bytes = 0;
}

int tc_check(tebd_handle *h) {
  if (!h->tc_err) return TEBD_OK;
  int e = 0;
  int rc = check_cuda(h, cudaMemcpyAsync(&e, h->tc_err, sizeof(int), cudaMemcpyDeviceToHost, h->stream),
                      "read tensor-core flag");
  if (rc) return rc;
  rc = check_cuda(h, cudaStreamSynchronize(h->stream), "read tensor-core flag");
  if (rc) return rc;
  if (e) {
    cudaMemsetAsync(h->tc_err, 0, sizeof(int), h->stream);
    return set_error(h, TEBD_ERR_CUDA, "a tensor-core pipeline wait timed out");
  }
  return TEBD_OK;
}

namespace {

// Power-of-two balance of the inner index for the default form: with a_g the largest
// |A(:, g)| and b_g the largest |B(g, :)|, A's column g is multiplied by 2^s and B's row by
// 2^-s so that both come near sqrt(a_g b_g).  The digits are cut off relative to the
// largest entry of a row of A and of a column of B; unbalanced, an inner index with
// small Lambda1 (Gamma1 ~ 1 / Lambda1 in a chain that is not left-canonical) costs every
// other one of them its low digits (energies of such a chain, span 6e-6: 7e-14 off
// instead of 2e-16; FP64 sums: 1.5e-15).  One warp per (bond, g); s goes to the slot's vn.
__global__ void __launch_bounds__(256) k_theta_balance(const double2 *__restrict__ gam, const double *__restrict__ lam,
                                                       const int *__restrict__ links, const Slot *slots, int chi,
                                                       int d) {
  const int s = blockIdx.y;
  const Compact cp = *slots[s].cp;
  const int gk = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (gk >= cp.r1) return;
  const int link = links[s], g = slots[s].idx1[gk];
  const size_t csz = (size_t)chi * d * chi;
  const double2 *G1 = gam + (size_t)(link - 1) * csz, *G2 = gam + (size_t)link * csz;
  const double *l0 = lam + (size_t)(link - 1) * chi, *l2 = lam + (size_t)(link + 1) * chi;
  const double l1 = lam[(size_t)link * chi + g];
  int ea = 0, eb = 0;  // largest exponent fields
  auto field = [](double x) { return (__double2hiint(x) >> 20) & 0x7ff; };
  for (int e = lane; e < d * cp.r0; e += 32) {
    const int i = e / cp.r0, a = slots[s].idx0[e - i * cp.r0];
    const double2 v = G1[a + (size_t)chi * i + (size_t)chi * d * g];
    ea = max(ea, max(field(v.x * l0[a]), field(v.y * l0[a])));
  }
  for (int e = lane; e < d * cp.r2; e += 32) {
    const int j = e / cp.r2, b = slots[s].idx2[e - j * cp.r2];
    const double2 v = G2[g + (size_t)chi * j + (size_t)chi * d * b];
    const double w = l1 * l2[b];
    eb = max(eb, max(field(v.x * w), field(v.y * w)));
  }
  ea = __reduce_max_sync(0xffffffffu, ea);
  eb = __reduce_max_sync(0xffffffffu, eb);
  if (lane == 0) reinterpret_cast<int *>(slots[s].vn)[gk] = ea && eb ? max(-500, min(500, (eb - ea) / 2)) : 0;
}

__global__ void __launch_bounds__(256) k_theta_operands(const double2 *__restrict__ gam,
                                                        const double *__restrict__ lam,
                                                        const int *__restrict__ links, const Slot *slots, int chi,
                                                        int d, int m_max, int r1_max, int n_max, int *status) {
  const int s = blockIdx.y;
  const Compact cp = *slots[s].cp;
  const int link = links[s];
  const size_t csz = (size_t)chi * d * chi;
  const double2 *G1 = gam + (size_t)(link - 1) * csz;
  const double2 *G2 = gam + (size_t)link * csz;
  const double *l0 = lam + (size_t)(link - 1) * chi;
  const double *l1 = lam + (size_t)link * chi;
  const double *l2 = lam + (size_t)(link + 1) * chi;
  const int *idx0 = slots[s].idx0, *idx1 = slots[s].idx1, *idx2 = slots[s].idx2;
  double2 *A = slots[s].aux;
  auto mark = [&](int q) {
    atomicOr(status, 1);
    atomicOr(&slots[q].cp->bad, 1);
  };
  double2 *B = A + (size_t)m_max * r1_max;
  const int *bal = reinterpret_cast<const int *>(slots[s].vn);  // with `status`: the default form
  auto pow2 = [](int k) { return __longlong_as_double((long long)(k + 1023) << 52); };
  const size_t na = (size_t)m_max * r1_max, total = na + (size_t)r1_max * n_max;
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < total; e += (size_t)gridDim.x * blockDim.x) {
    double2 v = make_double2(0.0, 0.0);
    if (e < na) {
      const int r = (int)(e % m_max), gk = (int)(e / m_max);
      if (r < cp.m && gk < cp.r1) {
        const int i = r / cp.r0, a = idx0[r - i * cp.r0], g = idx1[gk];
        v = cscale(G1[a + (size_t)chi * i + (size_t)chi * d * g], l0[a]);
        if (status) v = cscale(v, pow2(bal[gk]));
        if (status && !(isfinite(v.x) && isfinite(v.y))) mark(s);  // the digits of NaN and Inf are zeros
      }
      A[e] = v;
    } else {
      const size_t f = e - na;
      const int gk = (int)(f % r1_max), c = (int)(f / r1_max);
      if (gk < cp.r1 && c < cp.n) {
        const int j = c / cp.r2, b = idx2[c - j * cp.r2], g = idx1[gk];
        v = cscale(G2[g + (size_t)chi * j + (size_t)chi * d * b], l1[g] * l2[b]);
        if (status) v = cscale(v, pow2(-bal[gk]));
        if (status && !(isfinite(v.x) && isfinite(v.y))) mark(s);
      }
      B[f] = v;
    }
  }
}

}  // namespace

// Theta of the batch on the tensor cores; returns -1 (nothing launched) when a
// dimension of the batch is zero, the product is small or the default form has no memory for
// the digit planes, so that the caller forms it on the CUDA cores.
// The default form (0) takes this path for large products: 8 planes hold 56 bits below
// each row's and column's largest magnitude, so that the error of a sum of r1 products,
// about 2^-56 sqrt(r1) of the product of the two, is below FP64's own (640 x 128 x 640:
// 3e-17 against 1e-16 of the row and column maxima).  It is normwise per row and column:
// where a row's and a column's large factors lie at different inner indices the entry is
// small and FP64 would keep it to its own size.  The CUDA cores' kernel is bound by the
// FP64 pipe: 32 bonds of 640 x 640 (chi = 128) took 11.5 ms, 1.1 ms now, packs included.
int launch_theta_tc(tebd_handle *h, int nb) {
  int rc;
  const int form = h->theta_form ? h->theta_form : 100 + kOzMaxS;
  // the largest product that the batch can have: do not read the records for less
  if (!h->theta_form && (double)h->n * h->n * h->chi < kThetaTcMin) return -1;
  if ((rc = read_compaction(h, nb))) return rc;
  const std::vector<Compact> &cp = h->cps;
  int m_max = 0, n_max = 0, r1_max = 0;
  for (const Compact &c : cp) {
    m_max = std::max(m_max, c.m);
    n_max = std::max(n_max, c.n);
    r1_max = std::max(r1_max, c.r1);
  }
  // small products (early, low-rank updates) stay on the CUDA cores: packing and
  // the extra synchronisation cost more than the tiled FP64 kernel there
  if (m_max == 0 || n_max == 0 || r1_max == 0 || (double)m_max * n_max * r1_max < kThetaTcMin) return -1;
  const Slot &s0 = h->slots[0];
  const long long aux_stride = nb > 1 ? (long long)(h->slots[1].aux - s0.aux) : 0;
  ZProd z = {};
  z.a = s0.aux;
  z.a_stride = aux_stride;
  z.lda = m_max;
  z.b = s0.aux + (size_t)m_max * r1_max;
  z.b_stride = aux_stride;
  z.ldb = r1_max;
  z.nprob = nb;
  z.m = m_max;
  z.n = n_max;
  z.k = r1_max;
  z.form = form;
  z.rs = 1;
  z.cs = 0;  // column stride = the bond's own m
  z.m_d = &h->cp_d[0].m;
  z.n_d = &h->cp_d[0].n;
  z.dim_stride = (int)(sizeof(Compact) / sizeof(int));
  z.alpha = 1.0;
  z.optr = reinterpret_cast<const unsigned char *>(h->slots_d) + offsetof(Slot, X);
  z.optr_stride = (int)sizeof(Slot);
  if ((rc = tc_reserve(h, zprod_ws_bytes(z))))
    return h->theta_form || rc != TEBD_ERR_OOM ? rc : -1;  // the default form does without the digit planes
  const size_t total = (size_t)m_max * r1_max + (size_t)r1_max * n_max;
  unsigned gx = (unsigned)std::min<size_t>((total + 255) / 256, 2048);
  if (!h->theta_form) {
    k_theta_balance<<<dim3((r1_max + 7) / 8, nb), 256, 0, h->stream>>>(h->gam, h->lam, h->links_d, h->slots_d, h->chi,
                                                                      h->d);
    TEBD_LAUNCHED(h);
  }
  k_theta_operands<<<dim3(gx, nb), 256, 0, h->stream>>>(h->gam, h->lam, h->links_d, h->slots_d, h->chi, h->d,
                                                         m_max, r1_max, n_max,
                                                         h->theta_form ? nullptr : h->status_d);
  TEBD_LAUNCHED(h);
  tc_events(h, zprod_mma_flops(z, nb), &z.ev0, &z.ev1);
  if ((rc = check_cuda(h, zprod_run(z, h->tc_ws, h->tc_err, h->stream), "tensor-core Theta"))) return rc;
  h->launches += zprod_oz(z.form) ? 5 : 3;  // packs (+ exponent passes) and the product
  return TEBD_OK;
}

}  // namespace tebd

using namespace tebd;

extern "C" int tebd_set_theta_form(tebd_handle *h, int form) {
  if (!h) return TEBD_ERR_ARG;
  if (!(form == 0 || form == kTc3xTF32 || (form >= 103 && form <= 100 + kOzCallS)))
    return set_error(h, TEBD_ERR_ARG, "theta form must be 0, 3 (3xTF32) or 103..107 (bf16 digit planes)");
  if (h->mode != TEBD_MODE_DENSE && form != 0 && !zprod_oz(form))
    return set_error(h, TEBD_ERR_STATE, "NC handles take theta form 0 or 103..107 (3xTF32 is for dense handles)");
  h->theta_form = form;
  return TEBD_OK;
}
