// C-ABI tangent-linear and adjoint RK2 step, objective and checkpointed gradient.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <string>
#include <vector>

#include "gt_fft.cuh"
#include "gt_handle.h"
#include "gt_internal.h"

using namespace gt;
using namespace gtc;

// ===========================================================================
// Tangent-linear and adjoint RK2 step (the differentiation extension).
// With a the stage input, bc the Coriolis source and Q(a) = P invcurl
// fft_dir(u(a) x w(a)):  nlt(a; bc) = Q(a) + P invcurl(i omega kz bc).
//   TL:  dN = P invcurl[ fft_dir(du x w + u x dw) + i omega kz dbc ]
//   adjoint (inner products of gt_adjoint.cu): with mu = invcurl P lam and
//   g = fft_inv(mu):  lam_a = curl fft_dir(w x g) + k^2 fft_dir(g x u),
//   lam_bc = -i omega kz mu.
// The RK2 step and its zeroing of the k = 0 mode (rkstep.f90:44-48,
// 100-104) are differentiated on top.
// ===========================================================================
namespace {

struct F3 {
  void* p[3];
};

// The call's workspace: one block carved into groups of three fields.  A block
// of up to kKeep bytes stays with the handle for the next call (17 allocations and
// frees a call before; a tangent-linear and an adjoint step at 64 x 128 x 64 mixed
// went from 9.3 to 5.7 ms with this and the passes below), where a memory budget is
// set only what it leaves beside the handle's own estimate.
constexpr size_t kKeep = (size_t)2 << 30;

size_t keep_limit(const gt_handle* h) {
  uint64_t budget = 0;
  size_t own = 0;
  gt_get_memory_budget(&budget);
  if (budget == 0) return kKeep;
  gt_memory_estimate(&h->p, &own);
  return budget > own ? (size_t)std::min<uint64_t>(kKeep, budget - own) : 0;
}

template <typename R>
struct AdjWork {
  gt_handle* h;
  const DevTables<R>& tb;
  char* at = nullptr;
  size_t sbytes, rbytes;
  AdjWork(gt_handle* hh, const DevTables<R>& t) : h(hh), tb(t) {
    sbytes = h->g.field_elems() * sizeof(Cplx<R>);
    rbytes = (size_t)h->g.nx * h->g.ny * h->g.nz * sizeof(R);
  }
  ~AdjWork() {
    if (h->adj_bytes <= keep_limit(h)) return;
    cudaStreamSynchronize(h->stream);
    cudaFree(h->adj_mem);
    h->adj_mem = nullptr;
    h->adj_bytes = 0;
  }
  // Room for nspec spectral and nreal real groups.
  int reserve(size_t nspec, size_t nreal) {
    const size_t need = 3 * (nspec * sbytes + nreal * rbytes);
    if (h->adj_bytes < need) {
      CK(cudaStreamSynchronize(h->stream));
      if (h->adj_mem) cudaFree(h->adj_mem);
      h->adj_mem = nullptr;
      h->adj_bytes = 0;
      const cudaError_t e = cudaMalloc(&h->adj_mem, need);
      if (e != cudaSuccess) {
        h->adj_mem = nullptr;
        const int rc = cuda_fail(e, ("adjoint workspace of " + std::to_string(need) + " bytes").c_str());
        return e == cudaErrorMemoryAllocation ? GT_ENOMEM : rc;
      }
      h->adj_bytes = need;
    }
    at = static_cast<char*>(h->adj_mem);
    return GT_OK;
  }
  F3 group(bool real) {
    F3 f;
    for (int c = 0; c < 3; ++c, at += real ? rbytes : sbytes) f.p[c] = at;
    return f;
  }
  int fused(int op, const F3& out, const F3& a, const F3* b = nullptr, const F3* c = nullptr, const F3* o2 = nullptr,
            double f = 0, double kmin2 = 0) {
    CKI(launch_spec_fused<R>(h->g, tb, op, out.p, a.p, b ? b->p : nullptr, c ? c->p : nullptr, o2 ? o2->p : nullptr,
                             f, kmin2, h->stream));
    return GT_OK;
  }
  // u = C2R(curl a), w = C2R(k^2 a)
  int uw(const F3& a, const F3& u, const F3& w, int pruned) {
    CKI(launch_phys_uw<R>(h->g, tb, a.p, h->w, u.p, w.p, pruned, &h->pm, h->d_err, h->stream, hook_fn, h));
    return GT_OK;
  }
};

template <typename R>
struct StepCtx {
  AdjWork<R> W;
  F3 s[2], r[5], n1, c, t1, t2, t3;
  int pr;       // the states are zero outside the kept set
  static constexpr size_t kSpec = 7, kReal = 5;
  StepCtx(gt_handle* h, const DevTables<R>& tb) : W(h, tb), pr(use_pruning(h) ? 1 : 0) {}
  // `more` spectral groups beyond the step's own may be taken with W.group
  int init(size_t more) {
    const int rc = W.reserve(kSpec + more, kReal);
    if (rc) return rc;
    for (F3* f : {&s[0], &s[1], &n1, &c, &t1, &t2, &t3}) *f = W.group(false);
    for (F3& f : r) f = W.group(true);
    if (pr) CK(cudaMemsetAsync(n1.p[0], 0, 3 * W.sbytes, W.h->stream));   // only kept modes are written
    return GT_OK;
  }
  // dN = TL of nlt at (a; bc) in direction (da; dbc)
  int tl_nlt(const F3& a, const F3& da, const F3& dbc, const F3& dN) {
    gt_handle* h = W.h;
    int rc;
    if ((rc = W.uw(a, r[0], r[1], pr))) return rc;
    if ((rc = W.uw(da, r[2], r[3], 0))) return rc;
    CKI(launch_phys_cross<R>(h->g, 0, r[4].p, nullptr, r[0].p, r[1].p, r[2].p, r[3].p, h->stream));
    CKI(launch_fft_dir<R>(h->g, W.tb, r[4].p, s[0].p, 3, &h->pm, h->stream, hook_fn, h));
    return W.fused(kFuseTlTail, dN, s[0], &dbc);
  }
  // (lam_a, lam_bc) += adjoint of tl_nlt at (a; bc) applied to lam
  int adj_nlt(const F3& a, const F3& lam, const F3& lam_a, const F3& lam_bc) {
    gt_handle* h = W.h;
    int rc;
    if ((rc = W.fused(kFuseAdjHead, s[0], lam, nullptr, nullptr, &lam_bc))) return rc;   // mu
    CKI(launch_fft_inv<R>(h->g, W.tb, s[0].p, r[4].p, 3, h->p.truncate == 1 ? 1 : 0, &h->pm, h->stream, hook_fn,
                          h));   // g = C2R(mu), mu truncated
    if ((rc = W.uw(a, r[0], r[1], pr))) return rc;
    CKI(launch_phys_cross<R>(h->g, 1, r[2].p, r[3].p, r[0].p, r[1].p, r[4].p, nullptr, h->stream));   // w x g, g x u
    void* const real[6] = {r[2].p[0], r[2].p[1], r[2].p[2], r[3].p[0], r[3].p[1], r[3].p[2]};
    void* const spec[6] = {s[0].p[0], s[0].p[1], s[0].p[2], s[1].p[0], s[1].p[1], s[1].p[2]};
    CKI(launch_fft_dir<R>(h->g, W.tb, real, spec, 6, &h->pm, h->stream, hook_fn, h));
    return W.fused(kFuseAdjTail, lam_a, s[0], &lam_a, &s[1]);
  }
  // c = E(b + dt2 N1(b)), c(0) = 0, for the state b in the handle
  int stage(const F3& b) {
    CKI(nlt(W.h, b.p, b.p, n1.p, kNltOnly, pr));
    return W.fused(kFuseStage, c, b, &n1, nullptr, nullptr, W.tb.dt2);
  }
  // db' = TL of the RK2 step at b applied to db
  int tl(const F3& b, const F3& db, const F3& out) {
    int rc;
    if ((rc = stage(b))) return rc;
    if ((rc = tl_nlt(b, db, db, t1))) return rc;                                             // dN1
    if ((rc = W.fused(kFuseStage, t3, db, &t1, nullptr, nullptr, W.tb.dt2))) return rc;      // dc
    if ((rc = tl_nlt(c, t3, db, t1))) return rc;                                             // dN2
    return W.fused(kFuseTlEnd, out, db, &t1, nullptr, nullptr, W.tb.dt);
  }
  // lam = adjoint of the RK2 step at b applied to lam' (in: lp, out: out)
  int adj(const F3& b, const F3& lp, const F3& out) {
    int rc;
    if ((rc = stage(b))) return rc;
    // lam_N2 = dt E Z lam' (t2), lam_b = E E Z lam' (out)
    if ((rc = W.fused(kFuseAdjStart, t2, lp, nullptr, nullptr, &out, W.tb.dt))) return rc;
    CK(cudaMemsetAsync(t3.p[0], 0, 3 * W.sbytes, W.h->stream));
    if ((rc = adj_nlt(c, t2, t3, out))) return rc;                     // lam_c (t3), lam_b += lam_bc2
    // lam_b += E Z lam_c, lam_N1 = dt2 E Z lam_c (t2)
    if ((rc = W.fused(kFuseAdjMid, t2, t3, nullptr, nullptr, &out, W.tb.dt2))) return rc;
    return adj_nlt(b, t2, out, out);                                   // lam_b += lam_a1 + lam_bc1
  }
};

template <typename R>
const DevTables<R>& tables(gt_handle* h);
template <>
const DevTables<float>& tables<float>(gt_handle* h) { return h->t32; }
template <>
const DevTables<double>& tables<double>(gt_handle* h) { return h->t64; }

template <typename R>
int tl_or_adj(gt_handle* h, const double* in[3], double* out[3], bool adjoint) {
  StepCtx<R> S(h, tables<R>(h));
  int rc = S.init(2);
  if (rc) return rc;
  const F3 x = S.W.group(false), y = S.W.group(false);
  F3 b;
  for (int c = 0; c < 3; ++c) {
    if ((rc = upload_spec(h, in[c], x.p[c]))) return rc;
    CK(cudaStreamSynchronize(h->stream));
    b.p[c] = h->b[c];
  }
  rc = adjoint ? S.adj(b, x, y) : S.tl(b, x, y);
  if (rc) return rc;
  prefault(out, 3, spec_bytes(h->g));
  for (int c = 0; c < 3; ++c) {
    if ((rc = download_spec(h, y.p[c], out[c]))) return rc;
    CK(cudaStreamSynchronize(h->stream));
  }
  return check_device_flag(h);
}

// J = sum over stored modes with |k| >= kmin of fac |(curl b)_k|^2
template <typename R>
int objective(gt_handle* h, const F3& b, double kmin, double* J) {
  CKI(launch_shell_energy<R>(h->g, tables<R>(h), b.p, kmin * kmin, h->d_partials, h->npartials, h->d_result, h->stream));
  CK(cudaMemcpyAsync(h->h_result, h->d_result, sizeof(double), cudaMemcpyDeviceToHost, h->stream));
  CK(cudaStreamSynchronize(h->stream));
  *J = h->h_result[0];
  return GT_OK;
}

template <typename R>
int gradient(gt_handle* h, int nsteps, int32_t seed, int K, double kmin, double* J, double* gout[3]) {
  StepCtx<R> S(h, tables<R>(h));
  const size_t fb = S.W.sbytes;
  const int ncp = (nsteps - 1) / K + 1, nseg = std::min(K, nsteps);
  int rc = S.init((size_t)ncp + nseg + 3);
  if (rc) return rc;
  // checkpoints (state at steps 0, K, 2K, ...) and one segment of states
  std::vector<F3> cp(ncp), seg(nseg);
  for (auto& f : cp) f = S.W.group(false);
  for (auto& f : seg) f = S.W.group(false);
  const F3 b0 = S.W.group(false);
  F3 lam = S.W.group(false), lam2 = S.W.group(false), state;
  for (int c = 0; c < 3; ++c) {
    state.p[c] = h->b[c];
    CK(cudaMemcpyAsync(b0.p[c], h->b[c], fb, cudaMemcpyDeviceToDevice, h->stream));
  }
  const bool was_in_k = h->state_in_k;
  // the forcing realisation, drawn once and replayed in every recomputation
  std::vector<ForceEntry> all;
  std::vector<size_t> offs(1, 0);
  const bool forced = h->p.forcing != GT_FORCING_NONE && !h->ht.fix.empty();
  int32_t sd = seed;
  for (int k = 0; k < nsteps; ++k) {
    if (forced) draw_forcing(h->p, h->ht, sd, all);
    offs.push_back(all.size());
  }
  auto step_k = [&](int k) {
    std::vector<ForceEntry> e(all.begin() + offs[k], all.begin() + offs[k + 1]);
    std::vector<size_t> o = {0, e.size()};
    return run_steps(h, 1, e, o);
  };
  auto copy3 = [&](const F3& dst, const F3& src) {   // groups (and the handle's state) are contiguous
    cudaMemcpyAsync(dst.p[0], src.p[0], 3 * fb, cudaMemcpyDeviceToDevice, h->stream);
  };
  for (int k = 0; k < nsteps; ++k) {
    if (k % K == 0) copy3(cp[k / K], state);
    if ((rc = step_k(k))) return rc;
  }
  if ((rc = objective<R>(h, state, kmin, J))) return rc;
  // lam = dJ/db_n = curl(1_S curl b_n)
  if ((rc = S.W.fused(kFuseObj, lam, state, nullptr, nullptr, nullptr, 0, kmin * kmin))) return rc;
  for (int i = ncp - 1; i >= 0; --i) {
    const int k0 = i * K, k1 = nsteps - k0 < K ? nsteps : k0 + K;
    copy3(state, cp[i]);
    for (int k = k0; k < k1; ++k) {
      copy3(seg[k - k0], state);
      if (k + 1 < k1 && (rc = step_k(k))) return rc;
    }
    for (int k = k1 - 1; k >= k0; --k) {
      if ((rc = S.adj(seg[k - k0], lam, lam2))) return rc;
      std::swap(lam, lam2);
    }
  }
  copy3(state, b0);
  prefault(gout, 3, spec_bytes(h->g));
  CK(cudaStreamSynchronize(h->stream));
  h->state_in_k = was_in_k;
  for (int c = 0; c < 3; ++c) {
    if ((rc = download_spec(h, lam.p[c], gout[c]))) return rc;
    CK(cudaStreamSynchronize(h->stream));
  }
  return check_device_flag(h);
}

}  // namespace

extern "C" {

int gt_tl_step(gt_handle* h, const double* dbx, const double* dby, const double* dbz, double* ox,
               double* oy, double* oz) {
  if (!h || !dbx || !dby || !dbz || !ox || !oy || !oz) return GT_EINVAL;
  int rc = set_dev(h);
  if (rc) return rc;
  const double* in[3] = {dbx, dby, dbz};
  double* out[3] = {ox, oy, oz};
  return h->mixed ? tl_or_adj<float>(h, in, out, false) : tl_or_adj<double>(h, in, out, false);
}

int gt_adj_step(gt_handle* h, const double* lx, const double* ly, const double* lz, double* ox,
                double* oy, double* oz) {
  if (!h || !lx || !ly || !lz || !ox || !oy || !oz) return GT_EINVAL;
  int rc = set_dev(h);
  if (rc) return rc;
  const double* in[3] = {lx, ly, lz};
  double* out[3] = {ox, oy, oz};
  return h->mixed ? tl_or_adj<float>(h, in, out, true) : tl_or_adj<double>(h, in, out, true);
}

int gt_objective(gt_handle* h, double kmin, double* J) {
  if (!h || !J) return GT_EINVAL;
  int rc = set_dev(h);
  if (rc) return rc;
  F3 b;
  for (int c = 0; c < 3; ++c) b.p[c] = h->b[c];
  return h->mixed ? objective<float>(h, b, kmin, J) : objective<double>(h, b, kmin, J);
}

int gt_gradient(gt_handle* h, int32_t nsteps, int32_t seed, int32_t checkpoint_every, double kmin,
                double* J, double* gx, double* gy, double* gz) {
  if (!h || nsteps < 1 || checkpoint_every < 1 || !J || !gx || !gy || !gz) return GT_EINVAL;
  int rc = set_dev(h);
  if (rc) return rc;
  double* out[3] = {gx, gy, gz};
  return h->mixed ? gradient<float>(h, nsteps, seed, checkpoint_every, kmin, J, out)
                  : gradient<double>(h, nsteps, seed, checkpoint_every, kmin, J, out);
}

}  // extern "C"
