// Kernels of the FP64 form's passes in block fixed point (gt_fixed.cuh).
// Included by gt_kernels_impl.cuh for the double instantiation only.  The five
// passes are those of the header of gt_kernels_impl.cuh; fields b and c are
// FP64, the work fields hold longlong2 between the passes.
#pragma once

#include "gt_fixed.cuh"

namespace gt {

// Strided passes: 256 threads, tiles of 2048 / L columns (64-byte row segments
// at 512 points), so that every shared-memory offset is a compile-time one.
constexpr int kFxTileThreads = 256;
template <int LGL> constexpr int fx_tile() { return kFxTileThreads >> (LGL - 3); }
static inline int fx_lg_tile(int lgl) { return 11 - lgl; }

// Slots of a strided pass: lines are the tile's columns, x = threadIdx % TX.
template <int TX> using FxTileRed = FxRed<TX, 32, 1>;
template <int TX> __device__ __forceinline__ FxTileRed<TX> fx_red_tile(unsigned* slots, int x, int t) {
  return FxTileRed<TX>{slots, x & (kFxLines - 1), TX >= 32 || (int)(threadIdx.x & 31) < TX, t == 0};
}
// Slots of an x pass: lines are groups of T consecutive threads.
template <int LGN, int NQ> using FxRowRed = FxRed<1, ((1 << (LGN - 3)) < 32 ? (1 << (LGN - 3)) : 32), NQ>;
template <int LGN, int NQ> __device__ __forceinline__ FxRowRed<LGN, NQ> fx_red_rows(unsigned* slots, int grp, int t) {
  return FxRowRed<LGN, NQ>{slots, grp & (kFxLines - 1), (t & 31) == 0, t == 0};
}

// ---------------------------------------------------------------------------
// Pass 1: u = curl a, w = k^2 a in FP64, the six inverse z transforms in fixed
// point.  Each output line is formed from the input columns read again (after
// the first read, from L1 or L2), so a block needs one shared region and 24
// warps share an SM; with u_y and u_z parked in two more regions 16 do
// (1.99 against 1.91 ms at 512^3).  split: one output line per block
// (blockIdx.z = 6 member + line in a full launch, line in a pruned one), where
// the tiles alone leave SMs idle.
// ---------------------------------------------------------------------------
template <int LGZ>
__global__ void __launch_bounds__(kFxTileThreads, 3)
k_fx_zinv(Ptr6 a, Ptr6 w, DevTables<double> tb, Geom g, int pruned, const int32_t* __restrict__ tiles,
          int split, FxExp ex, long long fxs, long long mstride) {
  pass_enter();
  using C = double2;
  using E = longlong2;
  extern __shared__ __align__(16) unsigned char smraw[];
  constexpr int TX = fx_tile<LGZ>();
  __shared__ unsigned slots[FxTileRed<TX>::kSlots];
  __shared__ int emax[6][kFxLines];
  const int x = threadIdx.x % TX, t = threadIdx.x / TX;
  int tile = blockIdx.x, y = blockIdx.y;
  if (pruned) {
    tile = tiles[2 * blockIdx.x];
    y = tiles[2 * blockIdx.x + 1];
  }
  const unsigned mem = pruned ? blockIdx.y : (split ? blockIdx.z / 6 : blockIdx.z);
  const int f0 = split ? (int)(blockIdx.z % 6) : 0, f1 = split ? f0 + 1 : 6;
  const int X = tile * TX + x;
  const int ylim = pruned ? tb.xcut[y] : g.nh;
  const bool valid = X < ylim;
  constexpr int T = 1 << (LGZ - 3);
  const size_t plane = (size_t)g.ny * g.nhp;
  const size_t base = (size_t)y * g.nhp + (valid ? X : 0) + member_offset(mstride, mem);
  const int4* tw = reinterpret_cast<const int4*>(tb.fwz);
  auto red = fx_red_tile<TX>(slots, x, t);
  red.clear_all();
  for (int i = threadIdx.x; i < 6 * kFxLines; i += blockDim.x) (&emax[0][0])[i] = 0;
  __syncthreads();
  const double kx = valid ? tb.fkx[X] : 0.0, kxs = valid ? tb.fkxs[X] : 0.0;
  const double ky = tb.fky[y], kys = tb.fkys[y];
  const FxMem<LGZ, TX> mem_{reinterpret_cast<i64*>(smraw) + x};
  const size_t zstep = (size_t)T * plane;   // from a thread's position to its next
#pragma unroll 1
  for (int f = f0; f < f1; ++f) {
    // the fields output f reads: u_0 <- (a1, a2), u_1 <- (a2, a0), u_2 <- (a0, a1); w_c <- a_c.
    // u_f = i (k1 p2 - k2 p1) with (k1, k2) the wavenumbers of the two other axes in cyclic order
    const C* p1 = reinterpret_cast<const C*>(a.at(f < 3 ? (f == 2 ? 0 : f + 1) : f - 3));
    const C* p2 = reinterpret_cast<const C*>(a.at(f == 0 ? 2 : f - 1));
    C d[8];
    unsigned h = 0;
    p1 += base + (size_t)t * plane;
    p2 += base + (size_t)t * plane;
    const int32_t* cut = tb.xcut + (size_t)t * g.ny + y;
#pragma unroll
    for (int i = 0; i < 8; ++i, p1 += zstep, p2 += zstep, cut += T * g.ny) {
      const int z = t + i * T;
      const int lim = valid ? (pruned ? *cut : g.nh) : 0;
      d[i] = C{0, 0};
      if (X < lim) {
        const C q = *p1;
        if (f < 3) {
          const C r = *p2;
          const double kz = tb.fkz[z];
          const double k1 = f == 0 ? ky : (f == 1 ? kz : kx), k2 = f == 0 ? kz : (f == 1 ? kx : ky);
          d[i] = C{-k1 * r.y + k2 * q.y, k1 * r.x - k2 * q.x};   // produ.f90:44-63
        } else {
          const double k2 = (kxs + kys) + tb.fkzs[z];
          d[i] = C{k2 * q.x, k2 * q.y};
        }
        h = max(h, max(fx_abs_hi(d[i].x), fx_abs_hi(d[i].y)));
      }
    }
    int em = (int)(h >> 20);
    if constexpr (LGZ > 3) {
      em = (int)red.wmax((unsigned)em);
      if (red.lead) atomicMax(&emax[f][red.line], em);
      __syncthreads();
      em = emax[f][red.line];
    }
    E v[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = E{fx_from_double(d[i].x, em), fx_from_double(d[i].y, em)};
    int e = fx_exponent(em) + fx_line<+1>(v, t, tw, mem_, BlockSync{}, red);
    unsigned top = fx_top_put<LGZ>(red, fx_or_hi(v), 0);
    if constexpr (LGZ > 3) __syncthreads();
    top = fx_top_get<LGZ>(red, top, 0);
    red.par ^= 1;
    const int u = fx_headroom(top);
    E* out = reinterpret_cast<E*>(w.at(f)) + base + (size_t)t * plane;
    if (valid) {
#pragma unroll
      for (int i = 0; i < 8; ++i, out += zstep) *out = E{shl_clamp(v[i].x, u), shl_clamp(v[i].y, u)};
      if (t == 0) {
        if (e < kFxNaN / 2) e -= u;
        ex.ez[mem * fxs + ((size_t)f * g.ny + y) * g.nhp + X] = e;
        atomicMax(&ex.mz[mem * fxs + (size_t)f * g.nhp + X], e);
      }
    }
  }
}

// ---------------------------------------------------------------------------
// Strided transforms in place: KIND 0 the inverse y pass, 1 the forward y pass
// (both fixed point to fixed point), 2 a plain inverse z pass (FP64 in), 3 a
// plain forward z pass (FP64 out).  Blocks and masks are those of k_spass.
// ---------------------------------------------------------------------------
template <int KIND, int LGL>
__global__ void __launch_bounds__(kFxTileThreads, 3)
k_fx_spass(Ptr6 f, Geom g, const void* twv, long long ls, long long os, int xlim, int ymask,
           const int32_t* __restrict__ xcut0, int nf, FxExp ex, long long fxs, long long mstride) {
  pass_enter();
  using E = longlong2;
  constexpr int SIGN = (KIND == 0 || KIND == 2) ? +1 : -1;
  extern __shared__ __align__(16) unsigned char smraw[];
  constexpr int TX = fx_tile<LGL>();
  __shared__ unsigned slots[FxTileRed<TX>::kSlots];
  __shared__ int emax[KIND == 2 ? kFxLines : 1];
  const int x = threadIdx.x % TX, t = threadIdx.x / TX;
  const int X = blockIdx.x * TX + x;
  const int fi = blockIdx.z % nf, mem = blockIdx.z / nf, o = blockIdx.y;
  if (KIND == 2 && ymask == 3) {   // kept columns: X < xcut0[y]
    xlim = min(xlim, xcut0[o]);
    if ((int)blockIdx.x * TX >= xlim) return;
  }
  const bool valid = X < xlim;
  constexpr int T = 1 << (LGL - 3);
  E* p = reinterpret_cast<E*>(f.at(fi));
  const size_t base = (size_t)o * (size_t)os + (valid ? X : 0) + member_offset(mstride, mem);
  auto red = fx_red_tile<TX>(slots, x, t);
  red.clear_all();
  const long long xo = mem * fxs;
  const int Xc = valid ? X : 0;
  // element t of the line, and the step to t + T, t + 2 T, ...
  E* const p0 = p + base + (size_t)t * (size_t)ls;
  const size_t pstep = (size_t)T * (size_t)ls;
  E v[8];
  int e;
  if constexpr (KIND == 2) {
    double2 d[8];
    unsigned h = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      d[i] = valid ? reinterpret_cast<const double2*>(p0)[i * pstep] : double2{0, 0};
      h = max(h, max(fx_abs_hi(d[i].x), fx_abs_hi(d[i].y)));
    }
    int em = (int)(h >> 20);
    if constexpr (LGL > 3) {
      for (int i = threadIdx.x; i < kFxLines; i += blockDim.x) emax[i] = 0;
      __syncthreads();
      em = (int)red.wmax((unsigned)em);
      if (red.lead) atomicMax(&emax[red.line], em);
      __syncthreads();
      em = emax[red.line];
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = E{fx_from_double(d[i].x, em), fx_from_double(d[i].y, em)};
    e = fx_exponent(em);
  } else {
    // the largest exponent over the line's elements, and each element's own
    const int top = KIND == 0 ? ex.mz[xo + (size_t)fi * g.nhp + Xc]
                              : (KIND == 1 ? ex.mx[xo + (size_t)fi * g.nz + o] : ex.myf[xo + (size_t)fi * g.nhp + Xc]);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int r = t + i * T;
      const bool ld = valid && (ymask != 1 || X < xcut0[r]);
      const int* er = KIND == 0 ? ex.ez + xo + ((size_t)fi * g.ny + r) * g.nhp + Xc
                                : (KIND == 1 ? ex.ex + xo + ((size_t)fi * g.nz + o) * g.ny + r
                                             : ex.eyf + xo + ((size_t)fi * g.nz + r) * g.nhp + Xc);
      const int sh = top - (ld ? *er : 0) + (kFxOut - kFxIn);
      const E q = ld ? p[base + (size_t)r * (size_t)ls] : E{0, 0};
      // rounded where a line's integers may all be small: the rows of an x pass
      // have one exponent for all kx, and truncation's bias adds up in ky = 0
      const i64 half = KIND == 1 ? shl_clamp(1, sh - 1) : 0;
      v[i] = E{shr_clamp(q.x + half, sh), shr_clamp(q.y + half, sh)};
    }
    e = top >= kFxNaN / 2 ? kFxNaN : top + (kFxOut - kFxIn);
    if constexpr (LGL > 3) __syncthreads();   // the slots are clear
  }
  const FxMem<LGL, TX> mem_{reinterpret_cast<i64*>(smraw) + x};
  e += fx_line<SIGN>(v, t, reinterpret_cast<const int4*>(twv), mem_, BlockSync{}, red);
  if constexpr (KIND == 3) {
    if (valid) {
#pragma unroll
      for (int i = 0; i < 8; ++i)
        reinterpret_cast<double2*>(p0)[i * pstep] = double2{fx_to_double(v[i].x, e), fx_to_double(v[i].y, e)};
    }
  } else {
    unsigned mag = fx_top_put<LGL>(red, fx_or_hi(v), 0);
    if constexpr (LGL > 3) __syncthreads();
    mag = fx_top_get<LGL>(red, mag, 0);
    const int u = fx_headroom(mag);
    if (valid) {
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if (ymask != 2 || X < xcut0[t + i * T]) p0[i * pstep] = E{shl_clamp(v[i].x, u), shl_clamp(v[i].y, u)};
      if (t == 0) {
        if (e < kFxNaN / 2) e -= u;
        if constexpr (KIND == 0) {
          ex.ey[xo + ((size_t)fi * g.nz + o) * g.nhp + X] = e;
          atomicMax(&ex.my[xo + (size_t)fi * g.nz + o], e);
        } else if constexpr (KIND == 1) {
          ex.eyf[xo + ((size_t)fi * g.nz + o) * g.nhp + X] = e;
          atomicMax(&ex.myf[xo + (size_t)fi * g.nhp + X], e);
        } else {
          ex.ez[xo + ((size_t)fi * g.ny + o) * g.nhp + X] = e;
          atomicMax(&ex.mz[xo + (size_t)fi * g.nhp + X], e);
        }
      }
    }
  }
}

// ---------------------------------------------------------------------------
// Pass 3: per pair of rows the six C2R transforms, u x w and the three R2C
// transforms, all in fixed point.  Three groups of N/8 threads per pair: group q
// transforms the row's packed line q (fields 2 q, 2 q + 1) for both rows in
// turn, forms component q of u x w from the three lines in shared memory, and
// transforms that component of both rows forward as one complex line.  A thread
// holds one line's 8 values at a time, so 24 warps share an SM (one group per
// pair with its lines in registers: 12 warps and spills, 10.96 ms at 512^3).
// u and w of a row are brought to one exponent each (their largest components
// below 2^60), so u x w is limb products with 60 bits kept.
// ---------------------------------------------------------------------------
// (a b - c d) 2^-62, rounded; magnitudes below 2^60.
__device__ __forceinline__ i64 fx_det(const Limbs& a, const Limbs& b, const Limbs& c, const Limbs& d) {
  const i64 m1 = mad_wide(a.x0, b.x1, mad_wide(a.x1, b.x0, 1ll << 29));
  const i64 m2 = mad_wide(c.x0, d.x1, mad_wide(c.x1, d.x0, 0));
  return mad_wide(a.x1 << 2, b.x1, (m1 - m2) >> 30) - mad_wide(c.x1 << 2, d.x1, 0);
}

// The packed line position e = t + I N/8 of rows X1, X2 (pack_c2r_at) from
// fixed-point half spectra, each element shifted by its own exponent; the sum
// of two kFxIn - 1 bit values has kFxIn bits.
template <int I, int N>
__device__ __forceinline__ longlong2 fx_pack_c2r(const longlong2* __restrict__ X1, const longlong2* __restrict__ X2,
                                                 const int* __restrict__ e1, const int* __restrict__ e2, int top,
                                                 int t, int xa) {
  using E = longlong2;
  constexpr int T = N / 8, H = N / 2;
  const int k = I < 4 ? t + I * T : (I == 4 ? H - t : (8 - I) * T - t);
  if (k >= xa) return E{0, 0};
  const int base = top + (kFxOut - kFxIn + 1);
  E a = X1[k], b = X2[k];
  const int s1 = base - e1[k], s2 = base - e2[k];
  a.x = shr_clamp(a.x, s1);
  a.y = shr_clamp(a.y, s1);
  b.x = shr_clamp(b.x, s2);
  b.y = shr_clamp(b.y, s2);
  if constexpr (I == 0) {
    if (t == 0) { a.y = 0; b.y = 0; }
  }
  if constexpr (I == 4) {
    if (t == 0) return E{a.x, b.x};
  }
  if constexpr (I < 4) return E{a.x - b.y, a.y + b.x};
  return E{a.x + b.y, b.x - a.y};
}

// R2C split of a packed line kept in `mem`: entries k < xa of both half
// spectra, normalised by u; (a +- b)/2 is left to the exponent.
// SWAP: the line's real and imaginary parts are stored swapped.
template <bool SWAP, int LGN>
__device__ __forceinline__ void fx_split(const FxMem<LGN, 1>& mem, int t, int xa, int u, longlong2* oa, longlong2* ob) {
  constexpr int N = 1 << LGN, T = N / 8;
  for (int k = t; k < xa; k += T) {
    longlong2 a = mem.get(mem.at(k)), b = mem.get(mem.at((N - k) & (N - 1)));
    if (SWAP) {
      a = longlong2{a.y, a.x};
      b = longlong2{b.y, b.x};
    }
    oa[k] = longlong2{shl_clamp(a.x + b.x, u) >> 1, shl_clamp(a.y - b.y, u) >> 1};
    ob[k] = longlong2{shl_clamp(a.y + b.y, u) >> 1, shl_clamp(b.x - a.x, u) >> 1};
  }
}

template <int LGN> constexpr int fx_x_threads() { return LGN <= 8 ? 96 : 3 << (LGN - 3); }

template <int LGN>
__global__ void __launch_bounds__(fx_x_threads<LGN>(), 768 / fx_x_threads<LGN>())
k_fx_x(Ptr6 w, Geom g, const void* twv, int xa, int lgscale, FxExp ex, long long fxs, long long mstride) {
  pass_enter();
  using E = longlong2;
  extern __shared__ __align__(16) unsigned char smraw[];
  constexpr int N = 1 << LGN, T = N / 8, NQ = 2, LN = FxMem<LGN, 1>::kRows;
  __shared__ unsigned slots[FxRowRed<LGN, NQ>::kSlots];
  __shared__ unsigned bits[kFxLines][2];   // 8-point rows: the magnitudes of the line's two real rows
  __shared__ int expo[kFxLines];
  const int gid = threadIdx.x >> (LGN - 3), t = threadIdx.x & (T - 1);
  const int p = gid / 3, q = gid - 3 * p;   // row pair of the block, line of the row
  constexpr int P = fx_x_threads<LGN>() / (3 * T);
  const size_t pair = (size_t)blockIdx.x * P + p;
  const int4* tw = reinterpret_cast<const int4*>(twv);
  const size_t nhp = g.nhp;
  const size_t mo = member_offset(mstride, blockIdx.y);
  const long long xo = (long long)blockIdx.y * fxs;
  i64* const lines = reinterpret_cast<i64*>(smraw) + p * 6 * LN;   // three lines of two planes
  const FxMem<LGN, 1> mem{lines + q * 2 * LN};
  auto red = fx_red_rows<LGN, NQ>(slots, gid, t);
  red.clear_all();
  __syncthreads();
  const int z = (int)((2 * pair) >> g.lny), y0 = (int)((2 * pair) & (size_t)(g.ny - 1));
  // component q of u x w (produ.f90:14-16), u = (z0.x, z0.y, z1.x), w = (z1.y, z2.x, z2.y):
  // q = 0: uy wz - uz wy, 1: uz wx - ux wz, 2: ux wy - uy wx, as planes of the three lines
  const int c_u1 = LN * (q == 0 ? 1 : (q == 1 ? 2 : 0)), c_w1 = LN * (q == 0 ? 5 : (q == 1 ? 3 : 4));
  const int c_u2 = LN * (q == 0 ? 2 : (q == 1 ? 0 : 1)), c_w2 = LN * (q == 0 ? 4 : (q == 1 ? 5 : 3));
  E v[8];
  i64 c0[8];
  auto run = [&](auto sync) {
    int e = 0, ec0 = 0;
    // two rows to physical space and the product, then the component's two rows
    // forward: the same transform code each time (the forward one on swapped
    // real and imaginary parts), which keeps the kernel inside the instruction cache
#pragma unroll 1
    for (int r = 0; r < 3; ++r) {
      if (r < 2) {
        // line q: fields 2 q and 2 q + 1 of the row
        const size_t ro = mo + (2 * pair + r) * nhp;
        const E* X1 = reinterpret_cast<const E*>(w.at(2 * q)) + ro;
        const E* X2 = reinterpret_cast<const E*>(w.at(2 * q + 1)) + ro;
        const int* e1 = ex.ey + xo + ((size_t)(2 * q) * g.nz + z) * nhp;
        const int* e2 = e1 + (size_t)g.nz * nhp;
        const int top = max(ex.my[xo + (size_t)(2 * q) * g.nz + z], ex.my[xo + (size_t)(2 * q + 1) * g.nz + z]);
        for8([&](auto I) { v[I] = fx_pack_c2r<I, N>(X1, X2, e1, e2, top, t, xa); });
        e = top >= kFxNaN / 2 ? kFxNaN : top + (kFxOut - kFxIn + 1);
      }
      e += fx_line<+1>(v, t, tw, mem, sync, red);
      unsigned hx = 0, hy = 0;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        hx |= fx_abs_hi(v[i].x);
        hy |= fx_abs_hi(v[i].y);
      }
      mem.put_own(t, v);
      if (r == 2) {
        const unsigned mag = fx_top_put<LGN>(red, hx | hy, 0);
        sync();
        const int u = fx_headroom(fx_top_get<LGN>(red, mag, 0));
        E* out = reinterpret_cast<E*>(w.at(q)) + mo + (2 * pair) * nhp;
        fx_split<true>(mem, t, xa, u, out, out + nhp);
        if (t == 0) {
          if (e < kFxNaN / 2) e -= u + lgscale;
          int* eo = ex.ex + xo + ((size_t)q * g.nz + z) * g.ny + y0;
          eo[0] = e;
          eo[1] = e;
          atomicMax(&ex.mx[xo + (size_t)q * g.nz + z], e);
        }
        break;
      }
      hx = fx_top_put<LGN>(red, hx, 0);
      hy = fx_top_put<LGN>(red, hy, 1);
      if constexpr (LGN == 3) {
        bits[gid][0] = hx;
        bits[gid][1] = hy;
      }
      if (t == 0) expo[gid] = e;
      __syncthreads();   // the three lines of the row, their exponents and magnitudes
      // leading bit of line l's real (c = 0) or imaginary row
      auto lead = [&](int l, int c) {
        const unsigned h = LGN == 3 ? bits[3 * p + l][c] : *red.top(red.par, c, 3 * p + l);
        return expo[3 * p + l] + 64 - __clz((int)h);
      };
      // one exponent for u and one for w over the row; left shifts that take each component there
      const int eu = max(max(lead(0, 0), lead(0, 1)), lead(1, 0)) - 60;
      const int ew = max(max(lead(1, 1), lead(2, 0)), lead(2, 1)) - 60;
      const int e0 = expo[3 * p], e1 = expo[3 * p + 1], e2 = expo[3 * p + 2];
      int ec = max(max(e0, e1), e2) >= kFxNaN / 2 ? kFxNaN : eu + ew + 62;
      const int s_u1 = (q == 1 ? e1 : e0) - eu, s_w1 = (q == 1 ? e1 : e2) - ew;
      const int s_u2 = (q == 0 ? e1 : e0) - eu, s_w2 = (q == 2 ? e1 : e2) - ew;
      red.par ^= 1;
      const FxMem<LGN, 1> all{lines};
      auto product = [&](auto shift) {
        all.own(t, [&](int i, int o) {
          const i64* b = lines + o;
          const i64 c = fx_det(Limbs(shift(b[c_u1], s_u1)), Limbs(shift(b[c_w1], s_w1)), Limbs(shift(b[c_u2], s_u2)),
                               Limbs(shift(b[c_w2], s_w2)));
          if (r == 0) {
            c0[i] = c;
          } else {
            v[i] = E{c, c0[i]};   // swapped: c of row 0 is the real part
          }
        });
      };
      // right shifts only where a component is far below the others or fills its 61 bits
      if (min(min(s_u1, s_w1), min(s_u2, s_w2)) >= 0) {
        product([](i64 x, int n) { return shl_clamp(x, n); });
      } else {
        product([](i64 x, int n) { return n >= 0 ? shl_clamp(x, n) : shr_clamp(x, -n); });
      }
      if (r == 0) {
        ec0 = ec;
      } else {
        // the component's two rows as one line, at the larger exponent
        e = max(ec0, ec);
#pragma unroll
        for (int i = 0; i < 8; ++i) v[i] = E{shr_clamp(v[i].x, e - ec), shr_clamp(v[i].y, e - ec0)};
      }
      __syncthreads();   // everyone has read the lines
    }
  };
  if constexpr (T >= 32) {
    run(NamedSync{1 + gid, T});
  } else {
    run(BlockSync{});
  }
}

// Plain x transforms of one field (rows packed in pairs).
template <int LGN>
__global__ void __launch_bounds__(256)
k_fx_xc2r(Ptr6 specs, Ptr6 reals, Geom g, const void* twv, int P, int xa, FxExp ex) {
  pass_enter();
  using E = longlong2;
  extern __shared__ __align__(16) unsigned char smraw[];
  __shared__ unsigned slots[FxRowRed<LGN, 1>::kSlots];
  constexpr int N = 1 << LGN, lgT = LGN - 3, T = 1 << lgT, LN = FxMem<LGN, 1>::kRows;
  const int p = threadIdx.x >> lgT, t = threadIdx.x & (T - 1);
  const size_t pair = (size_t)blockIdx.x * P + p;
  const int f = blockIdx.y;   // field
  const E* X1 = reinterpret_cast<const E*>(specs.at(f)) + (2 * pair) * g.nhp;
  const E* X2 = X1 + g.nhp;
  double* real = reinterpret_cast<double*>(reals.at(f));
  const int z = (int)((2 * pair) >> g.lny);
  const int* e1 = ex.ey + ((size_t)f * g.nz + z) * g.nhp;   // both rows lie in plane z
  const int top = ex.my[(size_t)f * g.nz + z];
  auto red = fx_red_rows<LGN, 1>(slots, p, t);
  red.clear_all();
  E v[8];
  for8([&](auto I) { v[I] = fx_pack_c2r<I, N>(X1, X2, e1, e1, top, t, xa); });
  int e = top >= kFxNaN / 2 ? kFxNaN : top + (kFxOut - kFxIn + 1);
  __syncthreads();
  const FxMem<LGN, 1> mem{reinterpret_cast<i64*>(smraw) + p * 2 * LN};
  e += fx_line<+1>(v, t, reinterpret_cast<const int4*>(twv), mem, BlockSync{}, red);
  double* r0 = real + (2 * pair) * (size_t)N;
  double* r1 = r0 + N;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    r0[t + i * T] = fx_to_double(v[i].x, e);
    r1[t + i * T] = fx_to_double(v[i].y, e);
  }
}

template <int LGN>
__global__ void __launch_bounds__(256)
k_fx_xr2c(Ptr6 reals, Ptr6 specs, Geom g, const void* twv, int P, int lgscale, FxExp ex) {
  pass_enter();
  using E = longlong2;
  extern __shared__ __align__(16) unsigned char smraw[];
  __shared__ unsigned slots[FxRowRed<LGN, 1>::kSlots];
  __shared__ int emax[kFxLines];
  constexpr int N = 1 << LGN, lgT = LGN - 3, T = 1 << lgT, LN = FxMem<LGN, 1>::kRows;
  const int p = threadIdx.x >> lgT, t = threadIdx.x & (T - 1);
  const size_t pair = (size_t)blockIdx.x * P + p;
  const int f = blockIdx.y;   // field
  const double* r0 = reinterpret_cast<const double*>(reals.at(f)) + (2 * pair) * (size_t)N;
  const double* r1 = r0 + N;
  auto red = fx_red_rows<LGN, 1>(slots, p, t);
  red.clear_all();
  for (int i = threadIdx.x; i < kFxLines; i += blockDim.x) emax[i] = 0;
  double2 d[8];
  unsigned h = 0;
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    d[i] = double2{r0[t + i * T], r1[t + i * T]};
    h = max(h, max(fx_abs_hi(d[i].x), fx_abs_hi(d[i].y)));
  }
  __syncthreads();
  int em = (int)(h >> 20);
  if constexpr (LGN > 3) {
    em = (int)red.wmax((unsigned)em);
    if (red.lead) atomicMax(&emax[red.line], em);
    __syncthreads();
    em = emax[red.line];
  }
  E v[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) v[i] = E{fx_from_double(d[i].x, em), fx_from_double(d[i].y, em)};
  const FxMem<LGN, 1> mem{reinterpret_cast<i64*>(smraw) + p * 2 * LN};
  int e = fx_exponent(em) + fx_line<-1>(v, t, reinterpret_cast<const int4*>(twv), mem, BlockSync{}, red);
  mem.put_own(t, v);
  const unsigned mag = fx_top_put<LGN>(red, fx_or_hi(v), 0);
  __syncthreads();
  const int u = fx_headroom(fx_top_get<LGN>(red, mag, 0));
  E* spec = reinterpret_cast<E*>(specs.at(f));
  fx_split<false>(mem, t, g.nh, u, spec + (2 * pair) * (size_t)g.nhp, spec + (2 * pair + 1) * (size_t)g.nhp);
  if (t == 0) {
    if (e < kFxNaN / 2) e -= u + lgscale;
    int* eo = ex.ex + (size_t)f * g.nz * g.ny + 2 * pair;
    eo[0] = e;
    eo[1] = e;
    atomicMax(&ex.mx[(size_t)f * g.nz + ((2 * pair) >> g.lny)], e);
  }
}

// The spectral epilogue of pass 5 (nlt.f90:67-81, produ.f90:83-99,
// trunc.f90:14-28, rkstep.f90:30-48 / 86-104) at one thread's own positions, from
// the fixed-point transforms in three regions `reg` apart (exponents e).  The
// FP64 pipe bounds it, so with a = v + i omega kz b the update e (e' b + d i k x
// a / k^2) (e' = 1 or e) is formed with d k / k^2 as one vector, 1/k^2 comes from
// a table where the integrating factor does, and only the modes that are written
// are converted: 38 FP64 operations a mode instead of 61 with the division.  The
// increment is formed before the state is added, so that the state is rounded once (its
// two halves added to the state in turn left 19 % of the components a unit off after
// a step, for the same operations).
// (e' e as one factor would save six more, but its rounding repeats every step:
// 100 steps at 64^3 were off by 4.3e-15 instead of 0.9e-15.)
template <int LGT, int TX>
__device__ __forceinline__ void fx_epilogue(i64* __restrict__ sm, int reg, const int e[3], int t, int X, int y,
                                            int ylim, size_t base, size_t plane, const Ptr6& bc, const Ptr6& out,
                                            const DevTables<double>& tb, const Geom& g, int mode, int pruned) {
  using C = double2;
  constexpr int T = 1 << (LGT - 3);
  const double kx = tb.fkx[X], ky = tb.fky[y];
  const double kxys = tb.fkxs[X] + tb.fkys[y];
  const int k2xy = tb.emk_by_k2 ? (int)kxys : 0;
  const C* b0p = reinterpret_cast<const C*>(bc.p[0]);
  const C* b1p = reinterpret_cast<const C*>(bc.p[1]);
  const C* b2p = reinterpret_cast<const C*>(bc.p[2]);
  const FxMem<LGT, TX> mem{sm};
#pragma unroll 2
  for (int i = 0; i < 8; ++i) {
    const int z = t + i * T;
    const int zlim = tb.xcut[(size_t)z * g.ny + y];   // kept modes of this row: X < zlim
    if (X >= (pruned ? zlim : ylim)) continue;        // written columns: the kept ones, or all of the row's
    const size_t o = (size_t)z * plane + base;
    const C b0 = b0p[o], b1 = b1p[o], b2 = b2p[o];
    const int n = mem.at(z);
    const double kz = tb.fkz[z], okz = tb.omega * kz;
    const bool zero_mode = (X == 0) && (y == 0) && (z == 0);
    double em = 1.0, ik2;
    if (tb.emk_by_k2) {
      const int k2 = k2xy + (int)tb.fkzs[z];
      ik2 = tb.ik2[k2];
      if (mode != kNltOnly) em = tb.emk[k2];
    } else {
      ik2 = 1.0 / (kxys + tb.fkzs[z]);
      if (mode != kNltOnly) em = tb.emk[((size_t)z * g.ny + y) * g.nh + X];
    }
    auto val = [&](int f, const C& b) {   // v + i omega kz b(t)
      const longlong2 q = mem.get(n + f * reg);
      return C{fx_to_double(q.x, e[f]) - okz * b.y, fx_to_double(q.y, e[f]) + okz * b.x};
    };
    C a0 = val(0, b0), a1 = val(1, b1), a2 = val(2, b2);
    if (tb.truncate && (zero_mode || X >= zlim)) a0 = a1 = a2 = C{0, 0};
    C s0, s1, s2;
    if (mode == kNltOnly) {
      const double qx = kx * ik2, qy = ky * ik2, qz = kz * ik2;
      s0 = C{-qy * a2.y + qz * a1.y, qy * a2.x - qz * a1.x};
      s1 = C{-qz * a0.y + qx * a2.y, qz * a0.x - qx * a2.x};
      s2 = C{-qx * a1.y + qy * a0.y, qx * a1.x - qy * a0.x};
      if (zero_mode) { s0 = a0; s1 = a1; s2 = a2; }   // produ.f90:83
    } else {
      const double c = mode == kStage1 ? 1.0 : em;
      const double d = ik2 * (mode == kStage1 ? tb.dt2 : tb.dt);
      const double qx = kx * d, qy = ky * d, qz = kz * d;
      auto upd = [&](double b, double q1, double v1, double q2, double v2) {
        return em * fma(c, b, fma(q1, v1, -(q2 * v2)));
      };
      s0 = C{upd(b0.x, qz, a1.y, qy, a2.y), upd(b0.y, qy, a2.x, qz, a1.x)};
      s1 = C{upd(b1.x, qx, a2.y, qz, a0.y), upd(b1.y, qz, a0.x, qx, a2.x)};
      s2 = C{upd(b2.x, qy, a0.y, qx, a1.y), upd(b2.y, qx, a1.x, qy, a0.x)};
      if (zero_mode) s0 = s1 = s2 = C{0, 0};          // rkstep.f90:44-48 / 100-104
    }
    reinterpret_cast<C*>(out.p[0])[o] = s0;
    reinterpret_cast<C*>(out.p[1])[o] = s1;
    reinterpret_cast<C*>(out.p[2])[o] = s2;
  }
}

// ---------------------------------------------------------------------------
// Pass 5: forward z transforms in fixed point, then the FP64 epilogue at each
// thread's own positions.  Tiles and pruning are those of k_zfwd_epi.  TX: the
// tile width; a quarter of the usual one (blocks of 64 threads) where the usual
// tiles are fewer than two per SM, so that the epilogue's FP64 work spreads over
// all SMs.
// ---------------------------------------------------------------------------
template <int LGZ, int TX>
__global__ void __launch_bounds__(TX << (LGZ - 3), 512 / (TX << (LGZ - 3)))
k_fx_zfwd(Ptr6 w, Ptr6 bc, Ptr6 out, DevTables<double> tb, Geom g, int mode, int pruned,
          const int32_t* __restrict__ tiles, FxExp ex, long long fxs, Batch<double> bt) {
  pass_enter();
  using E = longlong2;
  extern __shared__ __align__(16) unsigned char smraw[];
  __shared__ unsigned slots[FxTileRed<TX>::kSlots];
  const int x = threadIdx.x % TX, t = threadIdx.x / TX;
  int tile = blockIdx.x, y = blockIdx.y;
  if (pruned) {
    tile = tiles[2 * blockIdx.x];
    y = tiles[2 * blockIdx.x + 1];
  }
  const int X = tile * TX + x;
  const int ylim = pruned ? tb.xcut[y] : g.nh;
  const bool valid = X < ylim;
  constexpr int T = 1 << (LGZ - 3);
  const size_t plane = (size_t)g.ny * g.nhp;
  const unsigned mem = pruned ? blockIdx.y : blockIdx.z;
  member_tables(bt, mem, tb);
  const size_t base = (size_t)y * g.nhp + (valid ? X : 0) + member_offset(bt.mstride, mem);
  constexpr int reg = FxMem<LGZ, TX>::kWords;
  const int4* tw = reinterpret_cast<const int4*>(tb.fwz);
  const long long xo = (long long)mem * fxs;
  auto red = fx_red_tile<TX>(slots, x, t);
  red.clear_all();
  __syncthreads();
  E v[8];
  int e[3];
#pragma unroll 1
  for (int f = 0; f < 3; ++f) {
    i64* S = reinterpret_cast<i64*>(smraw) + f * reg;
    const E* in = reinterpret_cast<const E*>(w.at(f)) + base + (size_t)t * plane;
    const int* er = ex.eyf + xo + ((size_t)f * g.nz + t) * g.nhp + (valid ? X : 0);
    const int top = ex.myf[xo + (size_t)f * g.nhp + (valid ? X : 0)];
#pragma unroll
    for (int i = 0; i < 8; ++i, in += (size_t)T * plane, er += T * g.nhp) {
      const int sh = top - (valid ? *er : 0) + (kFxOut - kFxIn);
      const E q = valid ? *in : E{0, 0};
      v[i] = E{shr_clamp(q.x, sh), shr_clamp(q.y, sh)};
    }
    const FxMem<LGZ, TX> mem_{S + x};
    int ef = top >= kFxNaN / 2 ? kFxNaN : top + (kFxOut - kFxIn);
    ef += fx_line<-1>(v, t, tw, mem_, BlockSync{}, red);
    red.par ^= 1;
    mem_.put_own(t, v);
    if (f == 0) e[0] = ef;
    if (f == 1) e[1] = ef;
    if (f == 2) e[2] = ef;
  }
  if (!valid) return;   // no barrier follows
  fx_epilogue<LGZ, TX>(reinterpret_cast<i64*>(smraw) + x, reg, e, t, X, y, ylim, base, plane, bc, out, tb, g, mode,
                       pruned);
}

}  // namespace gt
