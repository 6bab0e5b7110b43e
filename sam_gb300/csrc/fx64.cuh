// Fixed-point arithmetic of the FP64 line transforms.
//
// GB300 issues one FP64 instruction per 64 cycles and SM sub-partition, a
// 64-bit integer sum in 2 and a 32 x 32 -> 64-bit multiply-add in about 5
// (measured).  The transforms of the FP64 form therefore run in 64-bit fixed
// point on the integer pipes: a line's doubles become integers under one
// scale for the whole line, every butterfly sum is exact, every twiddle
// product is off by 2.5 units of the line's last place at most (below), and the
// results are converted back to doubles.
//
// Scale: with L1 = sum (|re| + |im|) over the line, every partial sum and
// every result of a discrete Fourier transform is at most L1 in modulus, so
// the line is scaled to L1 < 2^62 and nothing can overflow.  A unit in the
// last place is then at most 2^-61 L1 <= 2^-61 sqrt(2 n) |x|_2: about 2^-57
// of the line's norm at n = 256 and 2^-55.5 at n = 1024, which leaves room for
// the roundings of the twiddle products below the 2^-53 of FP64 arithmetic
// (tests/test_gpu_fixed_point.py and test_gpu_line_accuracy.py compare both
// with extended precision).
//
// Exceptional lines: a line holding an infinity or a NaN gives NaN
// throughout; lines whose largest value is so small or so large that the
// exponent arithmetic could leave the normal range take a slower exact path.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace samgpu {

__device__ __forceinline__ void team_sync(int TW);

// complex fixed-point value (units of the line's last place)
struct __align__(16) fxc {
  long long x, y;
};

// twiddle in units of 2^-62, each part split as h * 2^32 + l with l signed
struct __align__(16) fxw {
  int xh, xl, yh, yl;
};

__device__ __forceinline__ fxc cadd(fxc a, fxc b) { return fxc{a.x + b.x, a.y + b.y}; }
__device__ __forceinline__ fxc csub(fxc a, fxc b) { return fxc{a.x - b.x, a.y - b.y}; }

// h * 2^32 + l = v with l signed
struct FxSplit {
  int h, l;
};
__device__ __forceinline__ FxSplit fx_split(long long v) {
  return FxSplit{(int)((v + 0x80000000ll) >> 32), (int)v};
}
__host__ __device__ constexpr FxSplit fx_const(long long v) {
  return FxSplit{(int)((v + 0x80000000ll) >> 32), (int)(uint32_t)(v & 0xffffffffll)};
}
// (the instruction spelled out, so that it is the one intended)
__device__ __forceinline__ long long fx_mad(int a, int b, long long c) {
  long long r;
  asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(r) : "r"(a), "r"(b), "l"(c));
  return r;
}

// (A 2^32 + C) >> 30 for A the sum of the high products and C the cross terms
__device__ __forceinline__ long long fx_join(long long A, uint32_t clo) {
  const uint32_t lo = __funnelshift_l(clo, (uint32_t)A, 2);
  const uint32_t hi = __funnelshift_l((uint32_t)A, (uint32_t)(A >> 32), 2);
  return (long long)(((uint64_t)hi << 32) | lo);
}
// a * w, w in units of 2^-62, |w| <= 1: within 1.5 units (half of one by
// rounding, up to one by the low halves' product, which is left out)
__device__ __forceinline__ long long fx_mul(FxSplit a, FxSplit w) {
  const long long c = fx_mad(a.l, w.h, fx_mad(a.h, w.l, 1ll << 29));
  return fx_join(fx_mad(a.h, w.h, c >> 32), (uint32_t)c);
}
// the low halves' product, in units of the cross terms: added in products of
// fields (fx_mul_line), and with LOW in the twiddle products of the run-time
// path's long lines, whose units in the last place are coarser against their
// norm
__device__ __forceinline__ long long fx_low(FxSplit a, FxSplit w) { return (long long)__mulhi(a.l, w.l); }
// a * u + b * v, rounded once with LOW, else within 2.5 units.  (Without LOW a
// transform of 256 points is 0.35 x 2^-53 off instead of 0.31, of 512 0.80
// instead of 0.74: FP64 arithmetic 1.6-1.8.)  |a|, |b| < 2^62 with a^2 + b^2 < 2^124 and
// u^2 + v^2 <= 1 (or |a| + |b| < 2^62 and |u| + |v| < 1.6) keep the cross
// terms below 2^63.
template <bool LOW = false> __device__ __forceinline__ long long fx_dot(FxSplit a, FxSplit b, FxSplit u, FxSplit v) {
  long long c = fx_mad(b.l, v.h, fx_mad(b.h, v.l, fx_mad(a.l, u.h, fx_mad(a.h, u.l, 1ll << 29))));
  if (LOW) c += fx_low(a, u) + fx_low(b, v);
  return fx_join(fx_mad(b.h, v.h, fx_mad(a.h, u.h, c >> 32)), (uint32_t)c);
}
__device__ __forceinline__ FxSplit fx_neg(FxSplit w) { return FxSplit{-w.h, -w.l}; }

// a * w (SIGN = -1) or a * conj(w) (SIGN = +1)
template <int SIGN, bool LOW = false> __device__ __forceinline__ fxc ctw(fxc a, fxw w) {
  const FxSplit x = fx_split(a.x), y = fx_split(a.y), u{w.xh, w.xl}, v{w.yh, w.yl}, nv = fx_neg(v);
  if (SIGN < 0) return fxc{fx_dot<LOW>(x, y, u, nv), fx_dot<LOW>(x, y, v, u)};
  return fxc{fx_dot<LOW>(x, y, u, v), fx_dot<LOW>(x, y, nv, u)};
}
// a * (cr + i ci) for constants
__device__ __forceinline__ fxc fx_rot(fxc a, FxSplit cr, FxSplit ci) {
  const FxSplit x = fx_split(a.x), y = fx_split(a.y);
  return fxc{fx_dot(x, y, cr, fx_neg(ci)), fx_dot(x, y, ci, cr)};
}
template <int SIGN> __device__ __forceinline__ fxc cmul_si(fxc a) {
  return SIGN < 0 ? fxc{a.y, -a.x} : fxc{-a.y, a.x};
}
// constants of w9^J in units of 2^-62
constexpr long long kFxC9[5] = {0, 3532756447825785444ll, 800810873071977681ll, 0, -4333567320897763126ll};
constexpr long long kFxS9[5] = {0, 2964334632409774423ll, 4541624145405292212ll, 0, 1577289512995517789ll};
template <int SIGN, int J> __device__ __forceinline__ fxc rot9(fxc v) {
  return fx_rot(v, fx_const(kFxC9[J]), fx_const(SIGN * kFxS9[J]));
}
// v / 2, ties to even
__device__ __forceinline__ long long fx_half(long long v) { return (v + ((v >> 1) & 1)) >> 1; }
__device__ __forceinline__ long long fx_quarter(long long v) { return (v + 1 + ((v >> 2) & 1)) >> 2; }

// constants in units of 2^-62, rounded from extended precision
constexpr long long kFxH = 3260954456333195553ll;    // sqrt(2)/2
constexpr long long kFxC1 = 4260642322793532497ll;   // cos(pi/8)
constexpr long long kFxS1 = 1764815834521887442ll;   // sin(pi/8)
constexpr long long kFxS3 = 3993837246235628775ll;   // sin(2 pi/3)
constexpr long long kFxR5 = 2578010857022246787ll;   // sqrt(5)/4
constexpr long long kFxS51 = 4385974038932618941ll;  // sin(2 pi/5)
constexpr long long kFxS52 = 2710681029835013083ll;  // sin(4 pi/5)

template <int SIGN> __device__ __forceinline__ void dft8(fxc* a) {
  const FxSplit h = fx_const(kFxH);
  fxc b[8];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    b[q] = cadd(a[q], a[q + 4]);
    b[q + 4] = csub(a[q], a[q + 4]);
  }
  b[6] = cmul_si<SIGN>(b[6]);
  {
    // h (1 + SIGN i) and h (-1 + SIGN i)
    const long long p = b[5].x + b[5].y, m = b[5].x - b[5].y;
    b[5] = SIGN < 0 ? fxc{fx_mul(fx_split(p), h), fx_mul(fx_split(-m), h)}
                    : fxc{fx_mul(fx_split(m), h), fx_mul(fx_split(p), h)};
    const long long p7 = b[7].x + b[7].y, m7 = b[7].x - b[7].y;
    b[7] = SIGN < 0 ? fxc{fx_mul(fx_split(-m7), h), fx_mul(fx_split(-p7), h)}
                    : fxc{fx_mul(fx_split(-p7), h), fx_mul(fx_split(m7), h)};
  }
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    const fxc t0 = cadd(b[4 * e], b[4 * e + 2]), t1 = csub(b[4 * e], b[4 * e + 2]);
    const fxc t2 = cadd(b[4 * e + 1], b[4 * e + 3]), t3 = cmul_si<SIGN>(csub(b[4 * e + 1], b[4 * e + 3]));
    a[e] = cadd(t0, t2);
    a[4 + e] = csub(t0, t2);
    a[2 + e] = cadd(t1, t3);
    a[6 + e] = csub(t1, t3);
  }
}

template <int SIGN> __device__ __forceinline__ void dft3(fxc* a) {
  const FxSplit s = fx_const(SIGN * kFxS3);
  const fxc t = cadd(a[1], a[2]), d = csub(a[1], a[2]);
  const fxc m{a[0].x - fx_half(t.x), a[0].y - fx_half(t.y)};
  const fxc r{-fx_mul(fx_split(d.y), s), fx_mul(fx_split(d.x), s)};
  a[0] = cadd(a[0], t);
  a[1] = cadd(m, r);
  a[2] = csub(m, r);
}

// cos(2 pi/5), cos(4 pi/5) = -1/4 +- sqrt(5)/4
template <int SIGN> __device__ __forceinline__ void dft5(fxc* a) {
  const FxSplit r5 = fx_const(kFxR5), s1 = fx_const(SIGN * kFxS51), s2 = fx_const(SIGN * kFxS52);
  const fxc t1 = cadd(a[1], a[4]), d1 = csub(a[1], a[4]);
  const fxc t2 = cadd(a[2], a[3]), d2 = csub(a[2], a[3]);
  const fxc t = cadd(t1, t2), dt = csub(t1, t2);
  const fxc m{a[0].x - fx_quarter(t.x), a[0].y - fx_quarter(t.y)};
  const fxc c{fx_mul(fx_split(dt.x), r5), fx_mul(fx_split(dt.y), r5)};
  const fxc m1 = cadd(m, c), m2 = csub(m, c);
  const FxSplit x1 = fx_split(d1.x), y1 = fx_split(d1.y), x2 = fx_split(d2.x), y2 = fx_split(d2.y);
  const FxSplit ns1 = fx_neg(s1);
  const fxc n1{-fx_dot(y1, y2, s1, s2), fx_dot(x1, x2, s1, s2)};
  const fxc n2{-fx_dot(y1, y2, s2, ns1), fx_dot(x1, x2, s2, ns1)};
  a[0] = cadd(a[0], t);
  a[1] = cadd(m1, n1);
  a[4] = csub(m1, n1);
  a[2] = cadd(m2, n2);
  a[3] = csub(m2, n2);
}

// dft16 of fft_engine.cuh (4 x 4) with the rotations by odd multiples of
// pi/4 as a sum, a difference and two products
template <int SIGN> __device__ __forceinline__ void fx_dft4(fxc& a, fxc& b, fxc& c, fxc& d) {
  const fxc t0 = cadd(a, c), t1 = csub(a, c), t2 = cadd(b, d), t3 = cmul_si<SIGN>(csub(b, d));
  a = cadd(t0, t2);
  c = csub(t0, t2);
  b = cadd(t1, t3);
  d = csub(t1, t3);
}
template <int SIGN> __device__ __forceinline__ void dft16(fxc* a) {
  const FxSplit h = fx_const(kFxH);
#pragma unroll
  for (int n2 = 0; n2 < 4; ++n2) fx_dft4<SIGN>(a[n2], a[4 + n2], a[8 + n2], a[12 + n2]);
  // a[4 k1 + n2] *= w16^{n2 k1}
  auto rot = [&](fxc& v, long long cr, long long ci) { v = fx_rot(v, fx_const(cr), fx_const(SIGN * ci)); };
  auto rot45 = [&](fxc& v) {  // h (1 + SIGN i)
    const long long p = v.x + v.y, m = v.x - v.y;
    v = SIGN < 0 ? fxc{fx_mul(fx_split(p), h), fx_mul(fx_split(-m), h)}
                 : fxc{fx_mul(fx_split(m), h), fx_mul(fx_split(p), h)};
  };
  auto rot135 = [&](fxc& v) {  // h (-1 + SIGN i)
    const long long p = v.x + v.y, m = v.x - v.y;
    v = SIGN < 0 ? fxc{fx_mul(fx_split(-m), h), fx_mul(fx_split(-p), h)}
                 : fxc{fx_mul(fx_split(-p), h), fx_mul(fx_split(m), h)};
  };
  rot(a[4 + 1], kFxC1, kFxS1);
  rot45(a[8 + 1]);
  rot(a[12 + 1], kFxS1, kFxC1);
  rot45(a[4 + 2]);
  a[8 + 2] = cmul_si<SIGN>(a[8 + 2]);
  rot135(a[12 + 2]);
  rot(a[4 + 3], kFxS1, kFxC1);
  rot135(a[8 + 3]);
  rot(a[12 + 3], -kFxC1, -kFxS1);
#pragma unroll
  for (int k1 = 0; k1 < 4; ++k1) fx_dft4<SIGN>(a[4 * k1], a[4 * k1 + 1], a[4 * k1 + 2], a[4 * k1 + 3]);
  // a[4 k1 + k2] holds output k1 + 4 k2
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = i + 1; j < 4; ++j) {
      const fxc t = a[4 * i + j];
      a[4 * i + j] = a[4 * j + i];
      a[4 * j + i] = t;
    }
}

// ---------------------------------------------------------------- conversions
// The scale of a line: value = integer * 2^ex.
struct __align__(16) FxScale {
  int ex;
  int kind;    // kFxPlain, or one of the exceptional lines
  float norm;  // 2-norm of the transform's integers in units of 2^62 (where asked for)
};
constexpr int kFxPlain = 0;  // every result's exponent stays in the normal range
constexpr int kFxEdge = 1;   // it may not: results go through ldexp
constexpr int kFxNaN = 2;    // the line holds an infinity or a NaN
// lines whose largest value has a biased exponent below kFxTiny are lifted by
// 2^kFxLift before the conversion (subnormals become normal numbers)
constexpr int kFxTiny = 80, kFxLift = 256;

// Reduction over the TW threads of a team (all threads of the CTA call it).
// Teams of up to 32 threads lie within a warp, 32 / TW to a warp; wider ones
// are whole warps and go through shared memory.
template <typename V, typename Op> __device__ __forceinline__ V team_reduce(V v, int TW, Op op) {
  if (TW < 32 && (TW & (TW - 1))) {
    // not a power of two: folded onto the team's first lane, then broadcast
    const int lane = threadIdx.x & 31, tl = lane % TW, base = lane - tl;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      if (o >= TW) continue;
      const V t = __shfl_sync(0xffffffffu, v, (lane + o) & 31);
      if (tl < o && tl + o < TW && base + tl + o < 32) v = op(v, t);
    }
    return __shfl_sync(0xffffffffu, v, base);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
    if (o < TW) v = op(v, __shfl_xor_sync(0xffffffffu, v, o));
  if (TW > 32) {
    __shared__ V s_red[32];
    const int w = threadIdx.x >> 5, nw = TW >> 5, w0 = w & ~(nw - 1);
    if ((threadIdx.x & 31) == 0) s_red[w] = v;
    team_sync(TW);
    v = s_red[w0];
    for (int i = 1; i < nw; ++i) v = op(v, s_red[w0 + i]);
    team_sync(TW);
  }
  return v;
}

// largest |high word| of a thread's N values
template <int N> __device__ __forceinline__ uint32_t fx_max_hi(const double2* v) {
  uint32_t hm = 0;
#pragma unroll
  for (int i = 0; i < N; ++i)
    hm = max(hm, max((uint32_t)__double2hiint(v[i].x) & 0x7fffffffu, (uint32_t)__double2hiint(v[i].y) & 0x7fffffffu));
  return hm;
}
// sum of |v| / 2^(E - 1023) over a thread's N values from their leading 20
// bits: the high word less the exponent E, shifted into an FP32 pattern
template <int N> __device__ __forceinline__ float fx_l1(const double2* v, int E) {
  const int base = (E - 127) * (1 << 20);
  float s = 0.f, t = 0.f;
#pragma unroll
  for (int i = 0; i < N; ++i) {
    s += __int_as_float(max((__double2hiint(v[i].x) & 0x7fffffff) - base, 0) << 3);
    t += __int_as_float(max((__double2hiint(v[i].y) & 0x7fffffff) - base, 0) << 3);
  }
  return s + t;
}
// the double's mantissa as an integer with its leading bit at 62, shifted
// down by dsh less its biased exponent: cut off (only values too small for
// their last bits to reach the line's last place lose any), or, with NEAREST
// (the shift then is at least 1), rounded, ties to even
template <bool NEAREST = false> __device__ __forceinline__ long long fx_from(double d, int dsh) {
  const uint32_t hi = (uint32_t)__double2hiint(d), lo = (uint32_t)__double2loint(d);
  const int sh = dsh - (int)((hi >> 20) & 0x7ffu);
  const uint32_t mh = (__funnelshift_l(lo, hi, 10) & 0x3fffffffu) | 0x40000000u, ml = lo << 10;
  uint64_t m = ((uint64_t)mh << 32) | ml, rest = 0;
  // (shifts past 63 give 0)
  if (NEAREST) asm("shl.b64 %0, %1, %2;" : "=l"(rest) : "l"(m), "r"(64 - sh));
  asm("shr.u64 %0, %0, %1;" : "+l"(m) : "r"(sh));
  if (NEAREST) m += rest >= (1ull << 63) + (~m & 1);
  const long long s = (long long)((int)hi >> 31);
  return ((long long)m ^ s) - s;
}
// sum of (v / 2^(E - 1023))^2 from the same leading bits
template <int N> __device__ __forceinline__ float fx_l2(const double2* v, int E) {
  const int base = (E - 127) * (1 << 20);
  float s = 0.f, t = 0.f;
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const float x = __int_as_float(max((__double2hiint(v[i].x) & 0x7fffffff) - base, 0) << 3);
    const float y = __int_as_float(max((__double2hiint(v[i].y) & 0x7fffffff) - base, 0) << 3);
    s = fmaf(x, x, s);
    t = fmaf(y, y, t);
  }
  return s + t;
}
// The N values of each thread of a team to the line's fixed-point integers.
// NORM (lines whose transform becomes a product's factor; root_n = sqrt(n)):
// with the line's 2-norm, and scaled so that the transform's 2-norm, root_n
// times the line's, does not pass 2^62 either.
// NEAREST (lines of the run-time path, up to 1024 points): a line's unit in
// the last place grows with the square root of its length against its values,
// and beyond 512 points cutting those off was the largest error of a transform
// (white noise against extended precision, in units of 2^-53: 768 points 2.3
// cut off, 1.5 rounded; 1024 2.0 and 1.4; in FP64 arithmetic 1.9.  Rounding
// costs a step of 288^3 2.6 %).
template <int N, bool NORM, bool NEAREST = false> __device__ __forceinline__ FxScale fx_begin(double2* v, fxc* a, int TW, float root_n = 0.f) {
  const auto umax = [](uint32_t x, uint32_t y) { return max(x, y); };
  uint32_t hm = team_reduce(fx_max_hi<N>(v), TW, umax);
  FxScale sc{0, kFxPlain, 0.f};
  int lift = 0;
  if (hm < ((uint32_t)kFxTiny << 20) && hm > 0) {
    lift = kFxLift;
    const double f = __hiloint2double((1023 + kFxLift) << 20, 0);
    hm = 0;
#pragma unroll
    for (int i = 0; i < N; ++i) {
      v[i].x *= f;
      v[i].y *= f;
    }
    hm = fx_max_hi<N>(v);
  }
  if (__any_sync(0xffffffffu, lift)) hm = team_reduce(hm, TW, umax);
  const int E = (int)(hm >> 20);
  const auto sum = [](float x, float y) { return x + y; };
  float bound = team_reduce(fx_l1<N>(v, E), TW, sum), l2 = 0.f;
  if constexpr (NORM) {
    l2 = root_n * sqrtf(team_reduce(fx_l2<N>(v, E), TW, sum));
    bound = fmaxf(bound, l2);
  }
  // bound < 2^(E - 1023 + g) with room for the sums' own rounding
  int g = (__float_as_int(bound * 1.0001f) >> 23) - 126;
  if (E == 0) g = 128;  // a line of zeros
  if constexpr (NORM) sc.norm = l2 * __int_as_float(max(127 - g, 0) << 23);
  if (E == 0x7ff) sc.kind = kFxNaN;
  else if (lift || E + g > 2040) sc.kind = kFxEdge;
  sc.ex = E - 1023 - 62 + g - lift;
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const double2 d = v[i];
    a[i].x = fx_from<NEAREST>(d.x, E + g);
    a[i].y = fx_from<NEAREST>(d.y, E + g);
  }
  return sc;
}
// integer * 2^ex, rounded to nearest (kFxPlain: the exponent added in place)
__device__ __forceinline__ double fx_to(long long v, int ex) {
  const double r = __ll2double_rn(v);
  const int hi = __double2hiint(r);
  return __hiloint2double(hi ? hi + ex * (1 << 20) : 0, __double2loint(r));
}
// The same on the integer pipe, for kernels that the FP64 pipe bounds: the
// magnitude's leading one moved to bit 63, its top 53 bits rounded to
// nearest (halves away from zero).
__device__ __forceinline__ double fx_to_alu(long long v, int ex) {
  const long long s = v >> 63;
  const uint64_t m = (uint64_t)((v ^ s) - s);
  const int lz = __clzll((long long)m);
  const uint64_t t = m << lz;
  const uint64_t q = (t >> 11) + ((t >> 10) & 1);  // 2^52 .. 2^53
  const uint32_t hi = (uint32_t)(q >> 32) + (uint32_t)(1023 + 63 - 1 - lz + ex) * (1u << 20);
  return m ? __hiloint2double((int)(hi | ((uint32_t)(s >> 32) & 0x80000000u)), (int)(uint32_t)q) : 0.0;
}
// The parts' conversions: both on the FP64 pipe where the integer pipes are the
// bound (the transposes: 2-8 % slower otherwise), or, where a phase of the
// kernel does little else, one on each (x pass stores at 128^3 0.232 -> 0.220 ms,
// both on the integer pipe 0.222; at 256^3 1.074 -> 1.037, with a closure 3.08 ->
// 2.85, both on the integer pipe 3.09; z forward 0.863 -> 0.856).
enum FxConv { kFxOnFp64, kFxOnBoth };
template <FxConv CONV = kFxOnFp64> __device__ __forceinline__ double2 fx_out(fxc v, FxScale sc) {
  if (sc.kind == kFxPlain) {
    if (CONV == kFxOnBoth) return make_double2(fx_to(v.x, sc.ex), fx_to_alu(v.y, sc.ex));
    return make_double2(fx_to(v.x, sc.ex), fx_to(v.y, sc.ex));
  }
  if (sc.kind == kFxNaN) return make_double2(__hiloint2double(0x7ff80000, 0), __hiloint2double(0x7ff80000, 0));
  return make_double2(ldexp(__ll2double_rn(v.x), sc.ex), ldexp(__ll2double_rn(v.y), sc.ex));
}

// A line kept as split integers for products: value = (h 2^32 + l) 2^ex; norm
// <= 1 is the 2-norm of its integers, in units of 2^62.
struct __align__(16) FxLine {
  int ex, kind;
  float norm;
};
struct __align__(16) FxSplit2 {
  FxSplit x, y;
};
__device__ __forceinline__ FxSplit2 fx_split2(fxc v) { return FxSplit2{fx_split(v.x), fx_split(v.y)}; }
__device__ __forceinline__ fxc fx_whole(FxSplit2 v) {
  return fxc{v.x.h * (1ll << 32) + v.x.l, v.y.h * (1ll << 32) + v.y.l};
}

// The component-wise products of two lines (rhs.f's u_a u_b of two real rows
// at once) as one line's integers.  By Cauchy and Schwarz the sum of the
// products' moduli is at most the product of the lines' norms, so the 124-bit
// products shifted down by r = 62 + ceil(log2(norm_a norm_b)) sum to less
// than 2^62, the bound a transform needs; each is rounded once (all four
// products of halves are formed).
//
// With a subgrid term (a line of doubles whose moduli sum to less than
// 2^g.ex) both parts stay below 2^61: r grows by one, and further where the
// term is the larger part (down).
struct FxProduct {
  int s;  // 64 - r, at least 1 (norms up to 1) and at most 5 (lines scaled by their L1 norms have norms above 1/3)
  int down;
  long long half;
  FxScale sc;
};
__device__ __forceinline__ FxProduct fx_product(const FxLine& a, const FxLine& b, const FxLine* g = nullptr) {
  int r = min(max(62 + ((__float_as_int(a.norm * b.norm * 1.001f) >> 23) - 126), 59), 63);
  FxProduct p;
  if (g) r = max(r + 1, g->ex - 61 - a.ex - b.ex);
  p.sc.ex = a.ex + b.ex + r;
  p.down = min(max(r - 63, 0), 63);
  p.s = 64 - min(r, 63);
  p.half = 1ll << (31 - p.s);
  p.sc.norm = 0.f;
  // (room for the exponents of a scaling by 1 / (Nx Ny))
  p.sc.kind = (a.kind | b.kind | (g ? g->kind : 0)) & kFxNaN ? kFxNaN : (p.sc.ex < -960 || p.sc.ex > 940 ? kFxEdge : kFxPlain);
  return p;
}
// (with the low halves' product, up to 2^(62 - r) units: where a and b are the
// same field it is a square, and without it every product came out low, the
// mean of u u over 256 points by 0.5 x 2^-53 and over 1024 by 2.7 x 2^-53)
__device__ __forceinline__ long long fx_mul_line(FxSplit a, FxSplit b, const FxProduct& p) {
  const long long c = fx_mad(a.l, b.h, fx_mad(a.h, b.l, p.half + fx_low(a, b)));
  const long long A = fx_mad(a.h, b.h, c >> 32);
  const uint32_t lo = __funnelshift_l((uint32_t)c, (uint32_t)A, p.s);
  const uint32_t hi = __funnelshift_l((uint32_t)A, (uint32_t)(A >> 32), p.s);
  return (long long)(((uint64_t)hi << 32) | lo);
}
// a product of fx_mul_line joined with its subgrid term
__device__ __forceinline__ void fx_add_term(fxc& v, double2 t, const FxProduct& p) {
  const int dsh = p.sc.ex + 1023 + 62;
  v.x = (v.x >> p.down) + fx_from(t.x, dsh);
  v.y = (v.y >> p.down) + fx_from(t.y, dsh);
}
// The exponent bounding the moduli's sum of a line of n doubles (elements
// sidx(0) .. sidx(n - 1)), by one warp: sum < 2^info->ex.
__host__ __device__ __forceinline__ int sidx(int p);
__device__ __forceinline__ void fx_line_bound(const double2* line, FxLine* info, int n) {
  const int lane = threadIdx.x & 31;
  uint32_t hm = 0;
  for (int x = lane; x < n; x += 32) hm = max(hm, fx_max_hi<1>(line + sidx(x)));
  hm = __reduce_max_sync(0xffffffffu, hm);
  const int E = (int)(hm >> 20);
  float l1 = 0.f;
  for (int x = lane; x < n; x += 32) l1 += fx_l1<1>(line + sidx(x), E);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) l1 += __shfl_xor_sync(0xffffffffu, l1, o);
  const int g = (__float_as_int(l1 * 1.0001f) >> 23) - 126;
  if (lane == 0) *info = FxLine{E ? E - 1023 + g : -1100, E == 0x7ff ? kFxNaN : kFxPlain, 0.f};
}

}  // namespace samgpu
