// Block fixed-point line transforms: the FP64 form's FFTs on the integer pipe.
//
// GB300 issues 1.8 FP64 adds per clock and SM but 32 64-bit integer adds and
// 25-32 32x32+64-bit multiply-adds, so a line is transformed as 64-bit
// integers with one power-of-two scale per line instead of as doubles.  At
// 256^3 (ms a launch, FP64 arithmetic -> this): z inverse 0.93 -> 0.25, y inverse
// 1.54 -> 0.29, x 3.82 -> 0.83, y forward 0.77 -> 0.147, z forward 0.55 -> 0.197;
// the RK2 step 15.2 -> 3.40 ms, and 132.4 -> 25.0 ms at 512^3.  The x and y
// passes are bound by instruction issue (2.0-2.4 of 4 a clock) with the multiply
// pipe at 46-59 % and the ALU pipe at 50-57 %, DRAM at 12-35 %; the z passes also
// by their FP64 pointwise work (28-48 %) and spectral loads.
//
// * A line's inputs are scaled so that every component is below 2^59
//   (kFxIn bits); the first radix-8 stage adds at most 3.5 bits.
// * The sum over the line of |re| + |im| (its L1 norm) bounds every value any
//   later stage can produce, so a right shift chosen from that sum once keeps
//   all of them below 2^61: no value can overflow and no later stage has to look
//   at magnitudes.  Up to two of its bits wait until the last full radix-8
//   stage, where they are part of the twiddle product's own shift.
// * Twiddles are Q62; products are rounded to one unit.  The units lost are at
//   2^-61 of the line's L1 norm.  Relative L2 error of 3D transforms against
//   80-bit ones, FP64 arithmetic -> this: white noise 2.5e-16 -> 0.6-1.0e-16,
//   one mode over noise 2.0-3.8e-16 -> 0.5-1.0e-16, k^-5/3 fields 1.8-2.3e-16 ->
//   0.5-1.4e-16 (lines of 32 to 1024 points on each axis); the nonlinear term
//   3.0-3.5e-16 -> 1.3e-16.
// * Between passes a field stays fixed point: each pass normalises a line's
//   outputs to just below 2^61 and stores the line's exponent beside them
//   (value = integer * 2^exponent); the next pass, whose lines run across those
//   lines, shifts each element by its own exponent.  The largest exponent over
//   a next pass's line is kept by atomicMax as the lines are written.
// * A line that holds Inf or NaN gets the exponent kFxNaN, which survives every
//   maximum and comes out as NaN.  Inputs below 2^-1022 count as zero.
#pragma once

#include "gt_fft.cuh"

namespace gt {

constexpr int kFxIn = 59;        // bits of a line's scaled inputs
constexpr int kFxOut = 61;       // bits of stored values
constexpr int kFxNaN = 1 << 24;  // exponent of a line with a non-finite value

// ---- conversions ----------------------------------------------------------
__device__ __forceinline__ i64 shr_clamp(i64 x, int n) {   // n > 63 gives the sign
  i64 r;
  asm("shr.s64 %0, %1, %2;" : "=l"(r) : "l"(x), "r"(n));
  return r;
}
__device__ __forceinline__ i64 shl_clamp(i64 x, int n) {
  i64 r;
  asm("shl.b64 %0, %1, %2;" : "=l"(r) : "l"(x), "r"(n));
  return r;
}
// High word of |x|: its exponent field is bits 20..30.
__device__ __forceinline__ unsigned fx_abs_hi(double x) { return (unsigned)__double2hiint(x) & 0x7fffffffu; }

// x as a fixed-point integer of kFxIn bits, given the exponent field em of the
// line's largest value: value = result * 2^fx_exponent(em).
__device__ __forceinline__ i64 fx_from_double(double x, int em) {
  const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
  const int e = (int)((hi >> 20) & 0x7ffu);
  i64 m = (i64)(((unsigned long long)((hi & 0xfffffu) | 0x100000u) << 32) | lo) << (kFxIn - 53);
  m = shr_clamp(m, e ? em - e : 64);
  return (int)hi < 0 ? -m : m;
}
__device__ __forceinline__ int fx_exponent(int em) { return em >= 2047 ? kFxNaN : em - 1022 - kFxIn; }

// v * 2^e, rounded to nearest: the double's bits assembled with integer
// instructions (a conversion instruction issues at 2 per clock and SM).
__device__ __forceinline__ double fx_to_double(i64 v, int e) {
  const i64 s = v >> 63;
  const unsigned long long m = (unsigned long long)((v ^ s) - s);
  const int lz = __clzll((i64)m);
  unsigned long long q = ((m << lz) >> 1) + 0x200;        // 63 bits, the rounding bit added
  const int E = e + 1086 - lz;                            // exponent field of the result
  q >>= 10;                                               // implicit bit at 52 (or a carry to 53)
  unsigned hi = (unsigned)(q >> 32) + ((unsigned)(E - 1) << 20);
  unsigned lo = (unsigned)q;
  if (E >= 2047) { hi = 0x7ff00000u; lo = 0; }
  if (m == 0 || E <= 0) { hi = 0; lo = 0; }
  if (e >= kFxNaN / 2) { hi = 0x7ff80000u; lo = 0; }
  return __hiloint2double((int)(hi | ((unsigned)(s >> 32) & 0x80000000u)), (int)lo);
}
__device__ __forceinline__ unsigned fx_abs_hi(i64 v) { return (unsigned)abs((int)(v >> 32)); }

// ---- reductions over the threads of a line --------------------------------
// The line's threads in a warp are the lanes that differ in bits O0 <= 2^k < O1
// of the lane number (whole warps only); warps meet in shared slots.  Two slots
// per quantity and line, used in turn: a transform clears the other one between
// its own barriers, when everyone is done with it.
constexpr int kFxLines = 128;   // lines per block that need slots (lines of 16+ points)

template <int O0, int O1, int NQ> struct FxRed {
  unsigned* slots;   // sums [2][kFxLines], then magnitude bits [2][NQ][kFxLines]
  int line;
  bool lead;         // one lane per warp and line
  bool first;        // one thread per line
  int par = 0;
  static constexpr int kSlots = (2 + 2 * NQ) * kFxLines;

  __device__ __forceinline__ void clear_all() const {
    for (int i = threadIdx.x; i < kSlots; i += blockDim.x) slots[i] = 0;
  }
  __device__ __forceinline__ unsigned* sum(int p) const { return slots + p * kFxLines + line; }
  __device__ __forceinline__ unsigned* top(int p, int q, int l) const {
    return slots + (2 + p * NQ + q) * kFxLines + l;
  }
  __device__ __forceinline__ void clear_tops(int p) const {
#pragma unroll
    for (int q = 0; q < NQ; ++q) *top(p, q, line) = 0;
  }
  __device__ __forceinline__ unsigned wsum(unsigned v) const {
#pragma unroll
    for (int o = O0; o < O1; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
  }
  __device__ __forceinline__ unsigned wor(unsigned v) const {
#pragma unroll
    for (int o = O0; o < O1; o <<= 1) v |= __shfl_xor_sync(0xffffffffu, v, o);
    return v;
  }
  __device__ __forceinline__ unsigned wmax(unsigned v) const {
#pragma unroll
    for (int o = O0; o < O1; o <<= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
  }
};

// ---- the line transform ---------------------------------------------------
// Exchange scratch of TX interleaved lines (a strided tile's columns, or one x
// line): the real parts' plane, then the imaginary parts', one padding row after
// every 8: element e of the caller's line at (e + e / 8) TX of each plane.  Every
// access of a stage is one base plus a compile-time offset.
template <int LGL, int TX> struct FxMem {
  i64* s;   // the scratch plus the line's column
  static constexpr int T = 1 << (LGL - 3);
  static constexpr int kRows = strided_rows(1 << LGL);
  static constexpr int kPlane = kRows * TX;        // imaginary part of the element at s[o]: s[o + kPlane]
  static constexpr int kWords = 2 * kPlane;
  // position j of the radix-8 butterfly of thread t in the stage after 2^LGNS points
  template <int LGNS> __device__ __forceinline__ void put8(int t, const longlong2 v[8]) const {
    constexpr int step = LGNS == 0 ? TX : TX * ((1 << LGNS) + (1 << LGNS) / 8);
    const int e = ((t >> LGNS) << (LGNS + 3)) + (t & ((1 << LGNS) - 1));
    i64* const p = s + (LGNS == 0 ? 9 * TX * t : TX * (e + (e >> 3)));
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      p[j * step] = v[j].x;
      p[j * step + kPlane] = v[j].y;
    }
  }
  static __device__ __forceinline__ int at(int e) { return TX * (e + (e >> 3)); }
  // f(i, o) for this thread's positions t + i T, at s[o]
  template <typename F> __device__ __forceinline__ void own(int t, F&& f) const {
    if constexpr (T >= 8) {
      const int o = at(t);
#pragma unroll
      for (int i = 0; i < 8; ++i) f(i, o + i * TX * (T + T / 8));
    } else {
#pragma unroll
      for (int i = 0; i < 8; ++i) f(i, at(t + i * T));
    }
  }
  __device__ __forceinline__ longlong2 get(int o) const { return longlong2{s[o], s[o + kPlane]}; }
  __device__ __forceinline__ void put_own(int t, const longlong2 v[8]) const {
    own(t, [&](int i, int o) {
      s[o] = v[i].x;
      s[o + kPlane] = v[i].y;
    });
  }
};

// The stage that takes the delayed part f of the line's shift: the one after
// 64 points for lines of 512 and more (its inputs are sums of 64 of the line's,
// below 2^61 once 5 bits are gone), else the second one (sums of 8, 2 bits).
// Every rounding before it is then 2^f times smaller against the result:
// the error of a forward transform of a k^-5/3 field with 1024-point z lines goes
// from 2.0e-16 to 0.9e-16 (relative L2 against an 80-bit transform).
constexpr int fx_fold_stage(int lgl) { return lgl >= 9 ? 6 : 3; }
constexpr int fx_fold_need(int lgl) { return lgl >= 9 ? 5 : 2; }

template <int SIGN, int LGL, int LGNS, int TX, typename Sync>
__device__ __forceinline__ void fx_stages(longlong2 v[8], int t, const int4* __restrict__ tw,
                                          const FxMem<LGL, TX>& mem, const Sync& sync, int f) {
  constexpr int REM = LGL - LGNS, LR = REM >= 3 ? 3 : REM;
  constexpr int NS = 1 << LGNS, T = 1 << (LGL - 3);
  constexpr bool FOLD = LGNS == fx_fold_stage(LGL);
  const int4* tws = tw + (1 << LGL) + tw_stage_offset(LGL, LGNS);
  const i64 rnd = (1ll << 29) << (FOLD ? f : 0), half = FOLD ? (1ll << f) >> 1 : 0;
  auto mul = [&](longlong2& a, const int4* w) { a = twmul<SIGN>(a, __ldg(w), FOLD ? f : 0, rnd); };
  auto one = [&](longlong2& a) {   // an input without a twiddle
    if constexpr (FOLD) a = longlong2{shr_clamp(a.x + half, f), shr_clamp(a.y + half, f)};
  };
  if constexpr (LR == 3) {
    tws += t & (NS - 1);
    one(v[0]);
#pragma unroll
    for (int j = 1; j < 8; ++j) mul(v[j], &tws[(j - 1) * NS]);
    fx_dft8<SIGN>(v);
    if constexpr (REM > LR) {
      mem.template put8<LGNS>(t, v);
      sync();
      mem.own(t, [&](int i, int o) { v[i] = mem.get(o); });
      sync();
      fx_stages<SIGN, LGL, LGNS + LR, TX>(v, t, tw, mem, sync, f);
    }
  } else if constexpr (LR == 2) {
#pragma unroll
    for (int m = 0; m < 2; ++m) {
      const int4* q = tws + ((t + m * T) & (NS - 1));
      one(v[m]);
      mul(v[m + 2], q);
      mul(v[m + 4], q + NS);
      mul(v[m + 6], q + 2 * NS);
      fx_dft4<SIGN>(v[m], v[m + 2], v[m + 4], v[m + 6]);
    }
  } else if constexpr (LR == 1) {
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      one(v[m]);
      mul(v[m + 4], tws + ((t + m * T) & (NS - 1)));
      dft2(v[m], v[m + 4]);
    }
  }
}

__device__ __forceinline__ unsigned fx_or_hi(const longlong2 v[8]) {
  unsigned o = 0;
#pragma unroll
  for (int i = 0; i < 8; ++i) o |= fx_abs_hi(v[i].x) | fx_abs_hi(v[i].y);
  return o;
}

// v[i] = x[t + i L/8] scaled to kFxIn bits on entry, X[t + i L/8] * 2^-s on
// exit, |components| < 2^61.  Returns s.  The L1 sum is complete at the first
// exchange's barrier, so it costs none of its own.
template <int SIGN, int LGL, int TX, typename Sync, typename Red>
__device__ __forceinline__ int fx_line(longlong2 v[8], int t, const int4* __restrict__ tw,
                                       const FxMem<LGL, TX>& mem, const Sync& sync, const Red& red) {
  if constexpr (LGL == 3) {
    // one stage, a thread's own line: the shift its outputs need (0 to 2)
    fx_dft8<SIGN>(v);
    const int s = max(0, (64 - kFxOut) - __clz((int)fx_or_hi(v)));
    const i64 half = (1ll << s) >> 1;
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = longlong2{shr_clamp(v[i].x + half, s), shr_clamp(v[i].y + half, s)};
    return s;
  } else {
    // sum of the high words' magnitudes: up to 2^31 a thread; kept in units of 2^39
    unsigned acc = 16;
#pragma unroll
    for (int i = 0; i < 8; ++i) acc += fx_abs_hi(v[i].x) + fx_abs_hi(v[i].y);
    acc = red.wsum((acc >> 7) + 1);
    if (red.lead) atomicAdd(red.sum(red.par), acc);
    fx_dft8<SIGN>(v);
    mem.template put8<0>(t, v);
    sync();
    // L1 < (total + 8) 2^39 -> below 2^61 with 2^33 to spare for roundings
    const int s = max(0, 10 - __clz((int)(*red.sum(red.par) + 8u)));
    if (red.first) {
      *red.sum(red.par ^ 1) = 0;
      red.clear_tops(red.par ^ 1);
    }
    const int s1 = max(min(s, fx_fold_need(LGL)), s - 2);
    const i64 half = (1ll << s1) >> 1;
    mem.own(t, [&](int i, int o) {
      const longlong2 q = mem.get(o);
      v[i].x = shr_clamp(q.x + half, s1);
      v[i].y = shr_clamp(q.y + half, s1);
    });
    sync();
    fx_stages<SIGN, LGL, 3, TX>(v, t, tw, mem, sync, s - s1);
    return s;
  }
}

// Largest magnitude of quantity q over the line, as the OR of high words (its
// leading bit is the line's).  fx_top_put before a barrier, fx_top_get after.
template <int LGL, typename Red> __device__ __forceinline__ unsigned fx_top_put(const Red& red, unsigned v, int q) {
  if constexpr (LGL > 3) {
    v = red.wor(v);
    if (red.lead) atomicOr(red.top(red.par, q, red.line), v);
  }
  return v;
}
template <int LGL, typename Red> __device__ __forceinline__ unsigned fx_top_get(const Red& red, unsigned own, int q) {
  if constexpr (LGL > 3) return *red.top(red.par, q, red.line);
  return own;
}
// Left shift that brings magnitudes with high-word bits `top` to kFxOut bits
// (0 when they have them; values below 2^32 move by 29).
__device__ __forceinline__ int fx_headroom(unsigned top) { return max(0, __clz((int)top) - (64 - kFxOut)); }

// ---- exponents of the fixed-point work fields -----------------------------
// One int per line beside up to six work fields, in scratch the FP64 handle owns
// anyway (its transfer staging field, 4 nz ny nhp ints, which holds them for every
// grid of 8 points and more an axis).
struct FxExp {
  int* ez;    // [6][ny][nhp]  lines along z (inverse), by column (x, y)
  int* ey;    // [6][nz][nhp]  lines along y (inverse)
  int* ex;    // [6][nz][ny]   lines along x (forward)
  int* eyf;   // [6][nz][nhp]  lines along y (forward)
  int* mz;    // [6][nhp]      max of ez over y
  int* my;    // [6][nz]       max of ey over x
  int* mx;    // [6][nz]       max of ex over y
  int* myf;   // [6][nhp]      max of eyf over z
  size_t max_bytes;   // mz..myf, contiguous, set to kFxUnsetByte before the passes run
};
constexpr int kFxUnsetByte = 0x80;   // ints of -2139062144, below every exponent

static inline size_t fx_exp_ints(int ny, int nz, int nhp) {
  return (size_t)12 * nhp + (size_t)12 * nz + (size_t)6 * ny * nhp + (size_t)12 * nz * nhp + (size_t)6 * nz * ny;
}
static inline FxExp fx_exp(void* scratch, int ny, int nz, int nhp) {
  FxExp e;
  int* p = static_cast<int*>(scratch);
  auto take = [&](size_t n) { int* r = p; p += n; return r; };
  e.mz = take((size_t)6 * nhp);
  e.my = take((size_t)6 * nz);
  e.mx = take((size_t)6 * nz);
  e.myf = take((size_t)6 * nhp);
  e.max_bytes = ((size_t)12 * nhp + 12 * (size_t)nz) * sizeof(int);
  e.ez = take((size_t)6 * ny * nhp);
  e.ey = take((size_t)6 * nz * nhp);
  e.ex = take((size_t)6 * nz * ny);
  e.eyf = take((size_t)6 * nz * nhp);
  return e;
}

}  // namespace gt
