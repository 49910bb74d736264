// Building blocks of the tangent-linear and adjoint RK2 step: pointwise
// operators on groups of three spectral fields and on three real physical
// fields.  The step algebra itself is composed on the host (gt_tl_adj.cu).
//
// Inner products.  Spectral fields represent real fields; the adjoint is
// taken with respect to <x, y> = sum over stored modes of w_k Re(conj(x_k) y_k),
// w = 1 on the kx = 0 and kx = NX/2 planes and 2 elsewhere (the full-spectrum
// sum), and physical fields with sum_x f(x) g(x).  Under these, curl, k^2,
// invcurl, trunc and emk are self-adjoint, the Coriolis factor i omega kz has
// adjoint -i omega kz, fft_dir^T = fft_inv / (NX NY NZ) and
// fft_inv^T = (NX NY NZ) fft_dir.
#include <algorithm>

#include "gt_fft.cuh"
#include "gt_internal.h"

namespace gt {

namespace {

struct P3 {
  void* p[3];
};

// The step algebra's compound operators, one sweep each (a, b, c, o2 as named):
//  kFuseTlTail   : o = trunc invcurl (a + i omega kz b)
//  kFuseAdjHead  : o = invcurl trunc a, o2 += -i omega kz o
//  kFuseAdjTail  : o = b + curl a + k^2 c
//  kFuseStage    : o = Z E (a + f b)                     (Z: k = 0 mode to 0, E: emk)
//  kFuseTlEnd    : o = Z E (E a + f b)
//  kFuseAdjStart : o = f E Z a, o2 = E E Z a
//  kFuseAdjMid   : t = E Z a, o2 += t, o = f t
//  kFuseObj      : o = curl (1{|k| >= kmin} curl a)
template <typename R, int OP>
__global__ void __launch_bounds__(256)
k_spec_fused(P3 out, P3 a, P3 b, P3 c, P3 o2, DevTables<R> tb, Geom g, R f, R kmin2) {
  using C = Cplx<R>;
  const size_t rows = (size_t)g.ny * g.nz;
  // a warp walks a row
  const int lane = threadIdx.x & 31;
  for (size_t row = (size_t)blockIdx.x * 8 + (threadIdx.x >> 5); row < rows; row += (size_t)gridDim.x * 8) {
    const int y = (int)(row % g.ny), z = (int)(row / g.ny);
    const R ky = tb.fky[y], kz = tb.fkz[z];
    const int cut = tb.truncate ? tb.xcut[row] : g.nh;
    for (int X = lane; X < g.nh; X += 32) {
      const size_t o = row * g.nhp + X;
      auto ld = [&](const P3& p, C v[3]) {
        for (int q = 0; q < 3; ++q) v[q] = reinterpret_cast<const C*>(p.p[q])[o];
      };
      auto st = [&](const P3& p, const C v[3]) {
        for (int q = 0; q < 3; ++q) reinterpret_cast<C*>(p.p[q])[o] = v[q];
      };
      const R kx = tb.fkx[X];
      const R k2 = (tb.fkxs[X] + tb.fkys[y]) + tb.fkzs[z];
      const bool zero_mode = X == 0 && row == 0;
      const bool kill = tb.truncate && (zero_mode || X >= cut);
      auto curl = [&](const C v[3], R sc, C r[3]) {   // i sc k x v
        const R qx = sc * kx, qy = sc * ky, qz = sc * kz;
        r[0] = C{-qy * v[2].y + qz * v[1].y, qy * v[2].x - qz * v[1].x};
        r[1] = C{-qz * v[0].y + qx * v[2].y, qz * v[0].x - qx * v[2].x};
        r[2] = C{-qx * v[1].y + qy * v[0].y, qx * v[1].x - qy * v[0].x};
      };
      C va[3], r[3];
      if constexpr (OP == kFuseTlTail || OP == kFuseAdjHead) {
        for (int q = 0; q < 3; ++q) r[q] = C{0, 0};
        if (!kill) {
          ld(a, va);
          if constexpr (OP == kFuseTlTail) {
            C vb[3];
            ld(b, vb);
            const R okz = tb.omega * kz;
            for (int q = 0; q < 3; ++q) va[q] = C{va[q].x - okz * vb[q].y, va[q].y + okz * vb[q].x};
          }
          if (zero_mode) {
            for (int q = 0; q < 3; ++q) r[q] = va[q];
          } else {
            curl(va, (R)1 / k2, r);
          }
          if constexpr (OP == kFuseAdjHead) {
            C w[3];
            ld(o2, w);
            const R okz = tb.omega * kz;
            for (int q = 0; q < 3; ++q) w[q] = C{w[q].x + okz * r[q].y, w[q].y - okz * r[q].x};
            st(o2, w);
          }
        }
        st(out, r);
      } else if constexpr (OP == kFuseAdjTail) {
        C vb[3], vc[3];
        ld(a, va);
        ld(b, vb);
        ld(c, vc);
        curl(va, (R)1, r);
        for (int q = 0; q < 3; ++q) r[q] = C{(vb[q].x + r[q].x) + k2 * vc[q].x, (vb[q].y + r[q].y) + k2 * vc[q].y};
        st(out, r);
      } else if constexpr (OP == kFuseObj) {
        ld(a, va);
        C u[3];
        curl(va, (R)1, u);
        if (!(k2 >= kmin2)) u[0] = u[1] = u[2] = C{0, 0};
        curl(u, (R)1, r);
        st(out, r);
      } else {
        const R e = tb.emk_by_k2 ? tb.emk[(int)k2] : tb.emk[row * g.nh + X];
        ld(a, va);
        if constexpr (OP == kFuseStage || OP == kFuseTlEnd) {
          C vb[3];
          ld(b, vb);
          const R ea = OP == kFuseStage ? (R)1 : e;
          for (int q = 0; q < 3; ++q)
            r[q] = zero_mode ? C{0, 0} : C{e * (ea * va[q].x + f * vb[q].x), e * (ea * va[q].y + f * vb[q].y)};
          st(out, r);
        } else {
          C t[3], w[3];
          for (int q = 0; q < 3; ++q) {
            t[q] = zero_mode ? C{0, 0} : C{e * va[q].x, e * va[q].y};
            r[q] = C{f * t[q].x, f * t[q].y};
          }
          if constexpr (OP == kFuseAdjStart) {
            for (int q = 0; q < 3; ++q) w[q] = C{e * t[q].x, e * t[q].y};
          } else {
            ld(o2, w);
            for (int q = 0; q < 3; ++q) w[q] = C{t[q].x + w[q].x, t[q].y + w[q].y};
          }
          st(o2, w);
          st(out, r);
        }
      }
    }
  }
}

template <typename R> __device__ __forceinline__ void cross3(const R a[3], const R b[3], R r[3]) {
  r[0] = a[1] * b[2] - a[2] * b[1];
  r[1] = a[2] * b[0] - a[0] * b[2];
  r[2] = a[0] * b[1] - a[1] * b[0];
}

// Real fields.  ADJ false: o1 = c x b + a x d (du x w + u x dw for u, w, du, dw =
// a, b, c, d).  ADJ true: o1 = b x c, o2 = c x a (w x g and g x u for g = c).
template <typename R, bool ADJ>
__global__ void k_phys_cross(P3 o1, P3 o2, P3 a, P3 b, P3 c, P3 d, size_t n) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
    R u[3], w[3], x[3], y[3], r[3], q[3];
    for (int k = 0; k < 3; ++k) {
      u[k] = reinterpret_cast<const R*>(a.p[k])[i];
      w[k] = reinterpret_cast<const R*>(b.p[k])[i];
      x[k] = reinterpret_cast<const R*>(c.p[k])[i];
      if (!ADJ) y[k] = reinterpret_cast<const R*>(d.p[k])[i];
    }
    if constexpr (ADJ) {
      cross3(w, x, r);
      cross3(x, u, q);
    } else {
      cross3(x, w, r);
      cross3(u, y, q);
    }
    for (int k = 0; k < 3; ++k) {
      if constexpr (ADJ) {
        reinterpret_cast<R*>(o1.p[k])[i] = r[k];
        reinterpret_cast<R*>(o2.p[k])[i] = q[k];
      } else {
        reinterpret_cast<R*>(o1.p[k])[i] = r[k] + q[k];
      }
    }
  }
}

// partial[block] = the block's part of sum over modes with k2 >= kmin2 of
// fac |(curl b)|^2: the curl in the working precision, squares and sums in FP64;
// k_shell_sum adds the parts in order.
constexpr int kShellThreads = 256;
template <typename R>
__global__ void __launch_bounds__(kShellThreads)
k_shell_energy(P3 b, DevTables<R> tb, Geom g, R kmin2, double* partial) {
  using C = Cplx<R>;
  const size_t rows = (size_t)g.ny * g.nz;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double acc = 0.0;
  for (size_t row = (size_t)blockIdx.x * 8 + warp; row < rows; row += (size_t)gridDim.x * 8) {
    const int y = (int)(row % g.ny), z = (int)(row / g.ny);
    const R ky = tb.fky[y], kz = tb.fkz[z];
    for (int X = lane; X < g.nh; X += 32) {
      const R kx = tb.fkx[X];
      const R k2 = (tb.fkxs[X] + tb.fkys[y]) + tb.fkzs[z];
      if (!(k2 >= kmin2)) continue;
      const size_t o = row * g.nhp + X;
      const C v0 = reinterpret_cast<const C*>(b.p[0])[o], v1 = reinterpret_cast<const C*>(b.p[1])[o],
              v2 = reinterpret_cast<const C*>(b.p[2])[o];
      const double r0 = -ky * v2.y + kz * v1.y, i0 = ky * v2.x - kz * v1.x;
      const double r1 = -kz * v0.y + kx * v2.y, i1 = kz * v0.x - kx * v2.x;
      const double r2 = -kx * v1.y + ky * v0.y, i2 = kx * v1.x - ky * v0.x;
      const double fac = (X == 0 || X == g.nh - 1) ? 0.5 : 1.0;
      acc += fac * (((r0 * r0 + i0 * i0) + (r1 * r1 + i1 * i1)) + (r2 * r2 + i2 * i2));
    }
  }
  __shared__ double red[kShellThreads / 32];
  for (int off = 16; off > 0; off >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, off);
  if (lane == 0) red[warp] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0.0;
    for (int w = 0; w < kShellThreads / 32; ++w) s += red[w];
    partial[blockIdx.x] = s;
  }
}
__global__ void __launch_bounds__(256) k_shell_sum(double* partial, int n, double* out) {
  __shared__ double red[256];
  double s = 0.0;
  for (int i = threadIdx.x; i < n; i += 256) s += partial[i];
  red[threadIdx.x] = s;
  __syncthreads();
  for (int h = 128; h > 0; h >>= 1) {
    if ((int)threadIdx.x < h) red[threadIdx.x] += red[threadIdx.x + h];
    __syncthreads();
  }
  if (threadIdx.x == 0) *out = red[0];
}

P3 p3(void* const p[3], void* const fallback[3]) {
  P3 r;
  for (int c = 0; c < 3; ++c) r.p[c] = (p ? p : fallback)[c];
  return r;
}

}  // namespace

template <typename R>
int launch_spec_fused(const Geom& g, const DevTables<R>& tb, int op, void* const out[3], void* const a[3],
                      void* const b[3], void* const c[3], void* const o2[3], double f, double kmin2, void* stream) {
  const size_t rows = (size_t)g.ny * g.nz;
  const int blocks = (int)std::min<size_t>((rows + 7) / 8, 152 * 16);
  const P3 po = p3(out, out), pa = p3(a, a), pb = p3(b, a), pc = p3(c, a), p2 = p3(o2, out);
  switch (op) {
#define GT_OP(OP)                                                                                          \
  case OP:                                                                                                 \
    k_spec_fused<R, OP><<<blocks, 256, 0, (cudaStream_t)stream>>>(po, pa, pb, pc, p2, tb, g, (R)f, (R)kmin2); \
    break;
    GT_OP(kFuseTlTail) GT_OP(kFuseAdjHead) GT_OP(kFuseAdjTail) GT_OP(kFuseStage) GT_OP(kFuseTlEnd)
    GT_OP(kFuseAdjStart) GT_OP(kFuseAdjMid) GT_OP(kFuseObj)
#undef GT_OP
    default: return (int)cudaErrorInvalidValue;
  }
  return (int)cudaGetLastError();
}

template <typename R>
int launch_phys_cross(const Geom& g, int adjoint, void* const o1[3], void* const o2[3], void* const a[3],
                      void* const b[3], void* const c[3], void* const d[3], void* stream) {
  const size_t n = (size_t)g.nx * g.ny * g.nz;
  const int threads = 256;
  const int blocks = (int)std::min<size_t>((n + threads - 1) / threads, 152 * 16);
  const P3 po = p3(o1, o1), p2 = p3(o2, o1), pa = p3(a, a), pb = p3(b, a), pc = p3(c, a), pd = p3(d, a);
  if (adjoint)
    k_phys_cross<R, true><<<blocks, threads, 0, (cudaStream_t)stream>>>(po, p2, pa, pb, pc, pd, n);
  else
    k_phys_cross<R, false><<<blocks, threads, 0, (cudaStream_t)stream>>>(po, p2, pa, pb, pc, pd, n);
  return (int)cudaGetLastError();
}

template <typename R>
int launch_shell_energy(const Geom& g, const DevTables<R>& tb, void* const b[3], double kmin2, double* partials,
                        int cap, double* result, void* stream) {
  const size_t rows = (size_t)g.ny * g.nz;
  const int blocks = (int)std::min<size_t>((rows + 7) / 8, (size_t)std::min(cap, 152 * 8));
  k_shell_energy<R><<<blocks, kShellThreads, 0, (cudaStream_t)stream>>>(p3(b, b), tb, g, (R)kmin2, partials);
  k_shell_sum<<<1, 256, 0, (cudaStream_t)stream>>>(partials, blocks, result);
  return (int)cudaGetLastError();
}

#define GT_INST_ADJ(R)                                                                                             \
  template int launch_spec_fused<R>(const Geom&, const DevTables<R>&, int, void* const*, void* const*, void* const*, \
                                    void* const*, void* const*, double, double, void*);                            \
  template int launch_phys_cross<R>(const Geom&, int, void* const*, void* const*, void* const*, void* const*,      \
                                    void* const*, void* const*, void*);                                            \
  template int launch_shell_energy<R>(const Geom&, const DevTables<R>&, void* const*, double, double*, int, double*, \
                                      void*);
GT_INST_ADJ(float)
GT_INST_ADJ(double)

}  // namespace gt
