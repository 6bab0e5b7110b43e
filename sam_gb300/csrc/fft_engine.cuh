// Batched mixed-radix FFT engine for sm_103a: lines of length n <= 1024 held
// in shared memory, each line transformed by a team of threads.  A stage is a
// self-sorting Stockham step done in place: every thread first loads all of its
// butterfly inputs into registers, the team synchronises, then the thread
// computes and writes its outputs.
//  - Lengths of 8 to 256, and 512: radices (2 to 16), teams (of any width up to
//    a warp, packed into warps; 64 threads at 512) and every index but the
//    thread's place are fixed at compile time (ct_plan); at most 10 values a
//    thread.
//  - 256 points besides as 16 x 16 in registers (fft256_lines).
//  - The rest: radices 2, 3, 4, 5 and 8 read from the plan in shared memory,
//    teams of a power of two >= n / 8 threads (wider ones than a warp
//    synchronise on a named barrier), at most 8 values a thread.
// FP64 lines are integers under one scale while they are transformed (fx64.cuh).
//
// Conventions are FFTPACK's (the reference's fft.f): unnormalised transforms,
// SIGN = -1 is cfftf (exp(-i ...)), SIGN = +1 is cfftb (exp(+i ...)).
// Twiddles w_{l p}^{f q} are tabulated per stage (forward sign) by the host in
// extended precision and rounded once; the backward transform conjugates them.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

#include "fx64.cuh"

namespace samgpu {

template <typename T> struct Cx;
template <> struct Cx<double> { using type = double2; };
template <> struct Cx<float> { using type = float2; };
template <typename T> using cx_t = typename Cx<T>::type;

// Type of a transform's twiddles: fixed point for the FP64 form's lines
// (fx64.cuh), else the lines' own type.
template <typename C> struct TwOf { using type = C; };
template <> struct TwOf<double2> { using type = fxw; };
template <typename T> using tw_t = typename TwOf<cx_t<T>>::type;

template <typename C> __device__ __forceinline__ C mk(decltype(C::x) a, decltype(C::x) b) { C r; r.x = a; r.y = b; return r; }

template <typename C> __device__ __forceinline__ C cadd(C a, C b) { return mk<C>(a.x + b.x, a.y + b.y); }
template <typename C> __device__ __forceinline__ C csub(C a, C b) { return mk<C>(a.x - b.x, a.y - b.y); }
// FP32 complex sums as one packed instruction (add/sub.rn.f32x2: two IEEE
// round-to-nearest operations, the same results as the scalar pair)
__device__ __forceinline__ unsigned long long f2_pack(float2 a) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a.x), "f"(a.y));
  return r;
}
__device__ __forceinline__ float2 f2_unpack(unsigned long long r) {
  float2 a;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a.x), "=f"(a.y) : "l"(r));
  return a;
}
__device__ __forceinline__ float2 cadd(float2 a, float2 b) {
  unsigned long long r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(f2_pack(a)), "l"(f2_pack(b)));
  return f2_unpack(r);
}
__device__ __forceinline__ float2 csub(float2 a, float2 b) {
  unsigned long long r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(f2_pack(a)), "l"(f2_pack(b)));
  return f2_unpack(r);
}
// a * w (SIGN=-1) or a * conj(w) (SIGN=+1)
template <int SIGN, typename C> __device__ __forceinline__ C ctw(C a, C w) {
  if (SIGN < 0) return mk<C>(a.x * w.x - a.y * w.y, a.x * w.y + a.y * w.x);
  return mk<C>(a.x * w.x + a.y * w.y, a.y * w.x - a.x * w.y);
}
// FP32: the same products with their rounding spelled out (the second
// product rounded, the first fused with the sum), so every kernel computes
// the same bits whatever the compiler would contract at each call site
template <int SIGN> __device__ __forceinline__ float2 ctw(float2 a, float2 w) {
  if (SIGN < 0) return make_float2(__fmaf_rn(a.x, w.x, -__fmul_rn(a.y, w.y)), __fmaf_rn(a.x, w.y, __fmul_rn(a.y, w.x)));
  return make_float2(__fmaf_rn(a.x, w.x, __fmul_rn(a.y, w.y)), __fmaf_rn(a.y, w.x, -__fmul_rn(a.x, w.y)));
}
// multiply by SIGN * i  (exp(SIGN i pi/2))
template <int SIGN, typename C> __device__ __forceinline__ C cmul_si(C a) {
  if (SIGN < 0) return mk<C>(a.y, -a.x);
  return mk<C>(-a.y, a.x);
}

// Code paths of the line transforms: kFftAny picks at run time (the plan's
// length); kFft256 compiles only the 16 x 16 register path (n = 256) and
// kFftGeneric only the Stockham stages with the radix chosen at run time
// (kFftLong the same under another register budget);
// PATH = n (ct_length) compiles the Stockham stages of that length with their
// radices and every stride fixed at compile time (ct_plan).  A kernel built for one length
// thus carries no registers for another path.
constexpr int kFftAny = 0, kFft256 = 1, kFftGeneric = 2, kFftLong = 3;
// whether lines are transformed in fixed point (fx64.cuh)
template <typename C> inline constexpr bool kIsFx = std::is_same<C, double2>::value;

struct FftStage {
  int p;       // radix
  int l;       // length of the sub-transforms already combined
  int m;       // n / (l p)
  int tw_off;  // offset of this stage's l*(p-1) twiddles
  uint32_t mmul;  // exact b / m == (b * mmul) >> 21 for b < 2^11
};

struct FftPlan {
  int n;
  int nst;
  int tw_total;
  int team;     // threads per line of the run-time stages (at most 8 values per thread)
  int tw16_off; // n == 256: offset of the 16 x 16 table w_256^{f q} (else -1)
  int tw_pass;  // twiddles the pass kernels load: those of the length's own path (at 0), else all
  FftStage st[10];
};

// Values a thread holds per stage (8 complex: 16 in FP32 spills registers
// with five radices compiled into each stage loop).
template <typename C> struct Emax { static constexpr int value = 8; };

__device__ __forceinline__ int div_m(int b, const FftStage& s) { return (int)(((uint32_t)b * s.mmul) >> 21); }

// Shared-memory position of element p of a line: one pad slot after every 16
// elements, so the stride-16 row reads of the 16 x 16 path (and the strided
// reads of late Stockham stages) fall in distinct banks.
__host__ __device__ __forceinline__ int sidx(int p) { return p + (p >> 4); }
// Stride between consecutive lines: room for sidx(n - 1), rounded up to odd
// so lines start in rotating banks.
__host__ __device__ __forceinline__ int line_stride(int n) {
  const int s = n + ((n - 1) >> 4);
  return s | 1;
}

// Exact unsigned division by a runtime divisor d >= 1 for n < 2^31
// (round-up multiplier method): q = (umulhi(n, mul) + n) >> shift.
struct FastDiv {
  uint32_t d, mul, shift;
};
inline FastDiv make_fastdiv(uint32_t d) {
  FastDiv f;
  f.d = d;
  uint32_t s = 0;
  while ((1ull << s) < d) ++s;
  f.shift = s;
  f.mul = (uint32_t)(((1ull << 32) * ((1ull << s) - d)) / d + 1);
  return f;
}
__device__ __forceinline__ uint32_t fdiv(uint32_t n, const FastDiv& f) {
  return (uint32_t)(((uint64_t)__umulhi(n, f.mul) + n) >> f.shift);
}

// ---- radix-p DFT kernels on registers (in place on a[0..P-1])
template <int SIGN, typename C> __device__ __forceinline__ void dft2(C* a) {
  C t = a[1];
  a[1] = csub(a[0], t);
  a[0] = cadd(a[0], t);
}

template <int SIGN, typename C> __device__ __forceinline__ void dft4(C* a) {
  C t0 = cadd(a[0], a[2]), t1 = csub(a[0], a[2]);
  C t2 = cadd(a[1], a[3]), t3 = cmul_si<SIGN>(csub(a[1], a[3]));
  a[0] = cadd(t0, t2);
  a[2] = csub(t0, t2);
  a[1] = cadd(t1, t3);
  a[3] = csub(t1, t3);
}

template <int SIGN, typename C> __device__ __forceinline__ void dft8(C* a) {
  using T = decltype(C::x);
  const T h = (T)0.70710678118654752440084436210484903928;  // sqrt(2)/2
  // first level: pairs (q, q+4)
  C b0 = cadd(a[0], a[4]), b4 = csub(a[0], a[4]);
  C b1 = cadd(a[1], a[5]), b5 = csub(a[1], a[5]);
  C b2 = cadd(a[2], a[6]), b6 = csub(a[2], a[6]);
  C b3 = cadd(a[3], a[7]), b7 = csub(a[3], a[7]);
  // twiddles w8^{q} on the odd half: q=1 -> (1 + SIGN i) h, q=2 -> SIGN i, q=3 -> (-1 + SIGN i) h
  b6 = cmul_si<SIGN>(b6);
  {
    C t = b5;  // (t.x - SIGN? ) : multiply by h (1 + SIGN i)
    if (SIGN < 0) b5 = mk<C>((t.x + t.y) * h, (t.y - t.x) * h);
    else b5 = mk<C>((t.x - t.y) * h, (t.y + t.x) * h);
    t = b7;  // multiply by h (-1 + SIGN i)
    if (SIGN < 0) b7 = mk<C>((-t.x + t.y) * h, (-t.y - t.x) * h);
    else b7 = mk<C>((-t.x - t.y) * h, (-t.y + t.x) * h);
  }
  // two length-4 DFTs on (b0,b1,b2,b3) and (b4,b5,b6,b7)
  C e[4] = {b0, b1, b2, b3};
  C o[4] = {b4, b5, b6, b7};
  dft4<SIGN>(e);
  dft4<SIGN>(o);
  // outputs: even-indexed from e, odd-indexed from o
  a[0] = e[0]; a[2] = e[1]; a[4] = e[2]; a[6] = e[3];
  a[1] = o[0]; a[3] = o[1]; a[5] = o[2]; a[7] = o[3];
}

template <int SIGN, typename C> __device__ __forceinline__ void dft3(C* a) {
  using T = decltype(C::x);
  const T c1 = (T)-0.5;
  const T s1 = (T)SIGN * (T)0.86602540378443864676372317075293618347;  // SIGN*sin(2pi/3)
  C t = cadd(a[1], a[2]);
  C d = csub(a[1], a[2]);
  C y0 = cadd(a[0], t);
  C m = mk<C>(a[0].x + c1 * t.x, a[0].y + c1 * t.y);
  // SIGN i s * d
  C r = mk<C>(-s1 * d.y, s1 * d.x);
  a[0] = y0;
  a[1] = cadd(m, r);
  a[2] = csub(m, r);
}

template <int SIGN, typename C> __device__ __forceinline__ void dft5(C* a) {
  using T = decltype(C::x);
  const T c1 = (T)0.30901699437494742410229341718281905886;   // cos(2pi/5)
  const T c2 = (T)-0.80901699437494742410229341718281905886;  // cos(4pi/5)
  const T s1 = (T)SIGN * (T)0.95105651629515357211643933337938214340;  // sin(2pi/5)
  const T s2 = (T)SIGN * (T)0.58778525229247312916870595463907276860;  // sin(4pi/5)
  C t1 = cadd(a[1], a[4]), d1 = csub(a[1], a[4]);
  C t2 = cadd(a[2], a[3]), d2 = csub(a[2], a[3]);
  C y0 = cadd(a[0], cadd(t1, t2));
  C m1 = mk<C>(a[0].x + c1 * t1.x + c2 * t2.x, a[0].y + c1 * t1.y + c2 * t2.y);
  C m2 = mk<C>(a[0].x + c2 * t1.x + c1 * t2.x, a[0].y + c2 * t1.y + c1 * t2.y);
  // i*(s1 d1 + s2 d2) and i*(s2 d1 - s1 d2)
  C n1 = mk<C>(-(s1 * d1.y + s2 * d2.y), s1 * d1.x + s2 * d2.x);
  C n2 = mk<C>(-(s2 * d1.y - s1 * d2.y), s2 * d1.x - s1 * d2.x);
  a[0] = y0;
  a[1] = cadd(m1, n1);
  a[4] = csub(m1, n1);
  a[2] = cadd(m2, n2);
  a[3] = csub(m2, n2);
}

// v * (cr + i si) for real constants cr, si
template <typename C, typename T> __device__ __forceinline__ C crot(C v, T cr, T si) {
  return mk<C>(v.x * cr - v.y * si, v.x * si + v.y * cr);
}
__device__ __forceinline__ float2 crot(float2 v, float cr, float si) {
  return make_float2(__fmaf_rn(v.x, cr, -__fmul_rn(v.y, si)), __fmaf_rn(v.x, si, __fmul_rn(v.y, cr)));
}
// 16-point DFT in registers as 4 x 4: DFT4 over n1 of x[4 n1 + n2], the
// twiddles w16^{n2 k1}, DFT4 over n2; output k1 + 4 k2 in place.
template <int SIGN, typename C> __device__ __forceinline__ void dft16(C* a) {
  using T = decltype(C::x);
  const T c1 = (T)0.92387953251128675612818318939678828682;  // cos(pi/8)
  const T s1 = (T)0.38268343236508977172845998403039886676;  // sin(pi/8)
  const T h = (T)0.70710678118654752440084436210484903928;   // sqrt(2)/2
  C b[4][4];
#pragma unroll
  for (int n2 = 0; n2 < 4; ++n2) {
    C t[4] = {a[n2], a[4 + n2], a[8 + n2], a[12 + n2]};
    dft4<SIGN>(t);
#pragma unroll
    for (int k1 = 0; k1 < 4; ++k1) b[n2][k1] = t[k1];
  }
  // w16^j = (cos(2 pi j/16), SIGN sin(2 pi j/16)) for j = n2 k1
  auto rot = [&](C v, T cr, T si) { return crot(v, cr, si); };
  const T sg = (T)SIGN;
  b[1][1] = rot(b[1][1], c1, sg * s1);   // j = 1
  b[1][2] = rot(b[1][2], h, sg * h);     // j = 2
  b[1][3] = rot(b[1][3], s1, sg * c1);   // j = 3
  b[2][1] = rot(b[2][1], h, sg * h);     // j = 2
  b[2][2] = cmul_si<SIGN>(b[2][2]);      // j = 4
  b[2][3] = rot(b[2][3], -h, sg * h);    // j = 6
  b[3][1] = rot(b[3][1], s1, sg * c1);   // j = 3
  b[3][2] = rot(b[3][2], -h, sg * h);    // j = 6
  b[3][3] = rot(b[3][3], -c1, -sg * s1); // j = 9
#pragma unroll
  for (int k1 = 0; k1 < 4; ++k1) {
    C t[4] = {b[0][k1], b[1][k1], b[2][k1], b[3][k1]};
    dft4<SIGN>(t);
#pragma unroll
    for (int k2 = 0; k2 < 4; ++k2) a[k1 + 4 * k2] = t[k2];
  }
}

template <int P, int SIGN, typename C> __device__ __forceinline__ void dftp(C* a);
// times w9^J (exp(SIGN 2 pi i J / 9))
template <int SIGN, int J> __device__ __forceinline__ float2 rot9(float2 v) {
  constexpr double c[5] = {1.0, 0.76604444311897803520, 0.17364817766693034885, -0.5, -0.93969262078590838405};
  constexpr double s[5] = {0.0, 0.64278760968653932632, 0.98480775301220805937, 0.86602540378443864676, 0.34202014332566873304};
  return crot(v, (float)c[J], SIGN * (float)s[J]);
}
// N1 N2 points, coprime, without twiddles (Good and Thomas): input
// N2 n1 + N1 n2 (mod N) in row n1, column n2, output k in row k mod N1, column
// k mod N2
template <int N1, int N2, int SIGN, typename C> __device__ __forceinline__ void dft_coprime(C* a) {
  constexpr int N = N1 * N2;
  C t[N1][N2];
#pragma unroll
  for (int n2 = 0; n2 < N2; ++n2) {
    C c[N1];
#pragma unroll
    for (int n1 = 0; n1 < N1; ++n1) c[n1] = a[(N2 * n1 + N1 * n2) % N];
    dftp<N1, SIGN>(c);
#pragma unroll
    for (int n1 = 0; n1 < N1; ++n1) t[n1][n2] = c[n1];
  }
#pragma unroll
  for (int n1 = 0; n1 < N1; ++n1) dftp<N2, SIGN>(t[n1]);
#pragma unroll
  for (int k = 0; k < N; ++k) a[k] = t[k % N1][k % N2];
}
// 9 points as 3 x 3 with the twiddles w9^1, w9^2 (twice) and w9^4
template <int SIGN, typename C> __device__ __forceinline__ void dft9(C* a) {
  C b[3][3];
#pragma unroll
  for (int n2 = 0; n2 < 3; ++n2) {
    C c[3] = {a[n2], a[3 + n2], a[6 + n2]};
    dft3<SIGN>(c);
#pragma unroll
    for (int k1 = 0; k1 < 3; ++k1) b[n2][k1] = c[k1];
  }
  b[1][1] = rot9<SIGN, 1>(b[1][1]);
  b[1][2] = rot9<SIGN, 2>(b[1][2]);
  b[2][1] = rot9<SIGN, 2>(b[2][1]);
  b[2][2] = rot9<SIGN, 4>(b[2][2]);
#pragma unroll
  for (int k1 = 0; k1 < 3; ++k1) {
    C c[3] = {b[0][k1], b[1][k1], b[2][k1]};
    dft3<SIGN>(c);
#pragma unroll
    for (int k2 = 0; k2 < 3; ++k2) a[k1 + 3 * k2] = c[k2];
  }
}

template <int P, int SIGN, typename C> __device__ __forceinline__ void dftp(C* a) {
  if constexpr (P == 2) dft2<SIGN>(a);
  else if constexpr (P == 3) dft3<SIGN>(a);
  else if constexpr (P == 4) dft4<SIGN>(a);
  else if constexpr (P == 5) dft5<SIGN>(a);
  else if constexpr (P == 6) dft_coprime<2, 3, SIGN>(a);
  else if constexpr (P == 8) dft8<SIGN>(a);
  else if constexpr (P == 9) dft9<SIGN>(a);
  else if constexpr (P == 10) dft_coprime<2, 5, SIGN>(a);
  else if constexpr (P == 12) dft_coprime<3, 4, SIGN>(a);
  else if constexpr (P == 15) dft_coprime<3, 5, SIGN>(a);
  else dft16<SIGN>(a);
}

// One Stockham stage of radix P on one line held in shared memory.
// tl: lane index within the team, TW: team width.
__device__ __forceinline__ void team_sync(int TW) {
  if (TW <= 32) {
    __syncwarp();
  } else {
    const int id = 1 + (int)(threadIdx.x / TW);
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(TW) : "memory");
  }
}

// Reads element idx of the line being transformed (the stage's input).
template <typename C> struct LineLoad {
  const C* line;
  __device__ __forceinline__ C operator()(int idx) const { return line[sidx(idx)]; }
};

template <int P, int SIGN, typename C, typename Ld>
__device__ __forceinline__ void fft_stage(C* line, const C* __restrict__ tw, const FftStage& s, int n, int tl,
                                          int TW, Ld load) {
  constexpr int MAXB = Emax<C>::value / P;
  const int nb = n / P;
  C a[MAXB][P];
  int fo[MAXB], ko[MAXB];
#pragma unroll
  for (int i = 0; i < MAXB; ++i) {
    const int b = tl + i * TW;
    fo[i] = 0; ko[i] = 0;
    if (b < nb) {
      const int f = div_m(b, s);
      const int k = b - f * s.m;
      fo[i] = f; ko[i] = k;
      const int src = f * s.m * P + k;
      a[i][0] = load(src);
      if (s.l == 1) {
#pragma unroll
        for (int q = 1; q < P; ++q) a[i][q] = load(src + s.m * q);
      } else {
        const C* w = tw + s.tw_off + f * (P - 1);
#pragma unroll
        for (int q = 1; q < P; ++q) a[i][q] = ctw<SIGN>(load(src + s.m * q), w[q - 1]);
      }
    }
  }
  team_sync(TW);
#pragma unroll
  for (int i = 0; i < MAXB; ++i) {
    const int b = tl + i * TW;
    if (b < nb) {
      dftp<P, SIGN>(a[i]);
      const int dst = fo[i] * s.m + ko[i];
      const int os = s.l * s.m;
#pragma unroll
      for (int q = 0; q < P; ++q) line[sidx(dst + q * os)] = a[i][q];
    }
  }
  team_sync(TW);
}

// What becomes of the results of a fixed-point line: element idx, an integer
// of scale sc.  FxOutLine: doubles back into the line.
struct FxOutLine {
  static constexpr bool kNorm = false;
  double2* line;
  __device__ __forceinline__ void operator()(int idx, fxc v, FxScale sc) const { line[sidx(idx)] = fx_out(v, sc); }
};
// Doubles into the line, the band lo < idx < hi (which the caller does not
// read) left out.
struct FxOutBand {
  static constexpr bool kNorm = false;
  double2* line;
  int lo, hi;
  __device__ __forceinline__ void operator()(int idx, fxc v, FxScale sc) const {
    if (idx <= lo || idx >= hi) line[sidx(idx)] = fx_out(v, sc);
  }
};
// The integers into the line and their scale into *scale (the caller converts
// what it reads), or, with no scale given, doubles as FxOutLine.
struct FxOutInt {
  static constexpr bool kNorm = false;
  double2* line;
  FxScale* scale;
  __device__ __forceinline__ void operator()(int idx, fxc v, FxScale sc) const {
    if (scale) {
      reinterpret_cast<fxc*>(line)[sidx(idx)] = v;
      if (idx == 0) *scale = sc;
    } else {
      line[sidx(idx)] = fx_out(v, sc);
    }
  }
};
// Split integers for products and what fx_product needs to know of the line,
// or, with no info given, doubles.
struct FxOutSplit {
  static constexpr bool kNorm = true;
  double2* line;
  FxLine* info;
  __device__ __forceinline__ void operator()(int idx, fxc v, FxScale sc) const {
    if (info) {
      reinterpret_cast<FxSplit2*>(line)[sidx(idx)] = fx_split2(v);
      if (idx == 0) *info = FxLine{sc.ex, sc.kind, sc.norm};
    } else {
      line[sidx(idx)] = fx_out(v, sc);
    }
  }
};

// A first-stage loader that gives integers of a known scale (kInts) instead
// of doubles: a product line of two lines of split integers, plus the line g
// of doubles (a subgrid term; may be null).
struct FxProductLoad {
  static constexpr bool kInts = true;
  const FxSplit2 *a, *b;
  const double2* g;
  FxProduct p;
  __device__ __forceinline__ fxc operator()(int idx) const {
    const FxSplit2 ea = a[sidx(idx)], eb = b[sidx(idx)];
    fxc v{fx_mul_line(ea.x, eb.x, p), fx_mul_line(ea.y, eb.y, p)};
    if (g) fx_add_term(v, g[sidx(idx)], p);
    return v;
  }
  __device__ __forceinline__ FxScale scale() const { return p.sc; }
};
template <typename L, typename = void> struct LoadsInts { static constexpr bool value = false; };
template <typename L> struct LoadsInts<L, std::enable_if_t<L::kInts>> { static constexpr bool value = true; };

// The same stage of an FP64 line in fixed point (fx64.cuh).  The first stage
// (FIRST, l = 1: no twiddles) reads doubles through load and fixes the line's
// scale, which it leaves in sc; the others read the line's integers.  The
// last stage hands its results to out, the others write integers.
template <int P, int SIGN, bool FIRST, typename Ld, typename Out>
__device__ __forceinline__ void fx_stage(double2* line, const fxw* __restrict__ tw, const FftStage& s, int n, int tl,
                                         int TW, Ld load, Out out, FxScale& sc, bool last) {
  constexpr int MAXB = Emax<double2>::value / P;
  const int nb = n / P;
  fxc a[MAXB][P];
  int ds[MAXB];  // where the butterfly's outputs start
  if constexpr (FIRST && LoadsInts<Ld>::value) {
    sc = load.scale();
#pragma unroll
    for (int i = 0; i < MAXB; ++i) {
      const int b = tl + i * TW;
      ds[i] = b;
      if (b < nb) {
#pragma unroll
        for (int q = 0; q < P; ++q) a[i][q] = load(b + s.m * q);
      }
    }
  } else if constexpr (FIRST) {
    double2 v[MAXB][P];
#pragma unroll
    for (int i = 0; i < MAXB; ++i) {
      const int b = tl + i * TW;
      ds[i] = b;
#pragma unroll
      for (int q = 0; q < P; ++q) v[i][q] = make_double2(0.0, 0.0);
      if (b < nb) {
#pragma unroll
        for (int q = 0; q < P; ++q) v[i][q] = load(b + s.m * q);
      }
    }
    sc = fx_begin<MAXB * P, Out::kNorm, true>(&v[0][0], &a[0][0], TW, Out::kNorm ? sqrtf((float)n) : 0.f);
  } else {
    const fxc* fl = reinterpret_cast<const fxc*>(line);
#pragma unroll
    for (int i = 0; i < MAXB; ++i) {
      const int b = tl + i * TW;
      ds[i] = 0;
      if (b < nb) {
        const int f = div_m(b, s);
        const int src = b + f * s.m * (P - 1);
        ds[i] = b;
        const fxw* w = tw + s.tw_off + f * (P - 1);
        a[i][0] = fl[sidx(src)];
#pragma unroll
        for (int q = 1; q < P; ++q) a[i][q] = ctw<SIGN, true>(fl[sidx(src + s.m * q)], w[q - 1]);
      }
    }
  }
  team_sync(TW);
  const int os = s.l * s.m;
#pragma unroll
  for (int i = 0; i < MAXB; ++i) {
    const int b = tl + i * TW;
    if (b < nb) {
      dftp<P, SIGN>(a[i]);
      if (last) {
#pragma unroll
        for (int q = 0; q < P; ++q) out(ds[i] + q * os, a[i][q], sc);
      } else {
        fxc* fl = reinterpret_cast<fxc*>(line);
#pragma unroll
        for (int q = 0; q < P; ++q) fl[sidx(ds[i] + q * os)] = a[i][q];
      }
    }
  }
  team_sync(TW);
}
template <int SIGN, bool FIRST, typename Ld, typename Out>
__device__ __forceinline__ void fx_stage_p(double2* line, const fxw* __restrict__ tw, const FftStage& st, int n, int tl,
                                           int TW, Ld load, Out out, FxScale& sc, bool last) {
  switch (st.p) {
    case 8: fx_stage<8, SIGN, FIRST>(line, tw, st, n, tl, TW, load, out, sc, last); break;
    case 4: fx_stage<4, SIGN, FIRST>(line, tw, st, n, tl, TW, load, out, sc, last); break;
    case 2: fx_stage<2, SIGN, FIRST>(line, tw, st, n, tl, TW, load, out, sc, last); break;
    case 3: fx_stage<3, SIGN, FIRST>(line, tw, st, n, tl, TW, load, out, sc, last); break;
    default: fx_stage<5, SIGN, FIRST>(line, tw, st, n, tl, TW, load, out, sc, last); break;
  }
}

// Full transform of one line (all threads of the team call this together;
// a team with no line passes active=false and still synchronises).
template <int SIGN, typename C, typename Ld>
__device__ __forceinline__ void fft_stage_p(C* line, const C* __restrict__ tw, const FftStage& st, int n, int tl,
                                            int TW, Ld load) {
  switch (st.p) {
    case 8: fft_stage<8, SIGN>(line, tw, st, n, tl, TW, load); break;
    case 4: fft_stage<4, SIGN>(line, tw, st, n, tl, TW, load); break;
    case 2: fft_stage<2, SIGN>(line, tw, st, n, tl, TW, load); break;
    case 3: fft_stage<3, SIGN>(line, tw, st, n, tl, TW, load); break;
    default: fft_stage<5, SIGN>(line, tw, st, n, tl, TW, load); break;
  }
}

// Full transform of one line, the first stage reading its inputs through
// first(idx), so a caller can form the line on the fly (e.g. the product of
// two other lines).  All threads of the team call this together; a team with
// no line passes active=false and still synchronises.
template <int SIGN, typename C, typename First, typename Out>
__device__ __forceinline__ void fft_line_from(C* line, const typename TwOf<C>::type* __restrict__ tw, const FftPlan& pl,
                                              int tl, bool active, First first, Out out) {
  const int n = pl.n;
  const int TW = pl.team;
  const int tla = active ? tl : (1 << 20);  // inactive lanes own no butterfly
  if constexpr (kIsFx<C>) {
    FxScale sc;
    fx_stage_p<SIGN, true>(line, tw, pl.st[0], n, tla, TW, first, out, sc, pl.nst == 1);
    for (int s = 1; s < pl.nst; ++s)
      fx_stage_p<SIGN, false>(line, tw, pl.st[s], n, tla, TW, LineLoad<C>{line}, out, sc, s + 1 == pl.nst);
  } else {
    fft_stage_p<SIGN>(line, tw, pl.st[0], n, tla, TW, first);
    for (int s = 1; s < pl.nst; ++s) fft_stage_p<SIGN>(line, tw, pl.st[s], n, tla, TW, LineLoad<C>{line});
  }
}

// n = 256 as 16 x 16 in registers: a team of 16 threads per line, two lines
// per warp.  Thread k first transforms the column x[k + 16 q] (the l = 1
// Stockham stage of radix 16) and writes it back; thread f then reads row
// 16 f + q, applies w_256^{f q} and transforms it (the l = 16 stage).  One
// shared-memory exchange and four warp barriers per line.
template <int SIGN, typename C, typename First, typename Out>
__device__ __forceinline__ void fft256_lines(C* base, int ld, int nlines, const C* __restrict__ tw,
                                             const FftPlan& pl, First first, Out) {
  const int team = threadIdx.x >> 4;
  const int k = threadIdx.x & 15;
  const int nteams = blockDim.x >> 4;
  const int rounds = (nlines + nteams - 1) / nteams;
  const C* w = tw + pl.tw16_off + k;  // w[16 q] = w_256^{k q}
  for (int r = 0; r < rounds; ++r) {
    const int L = r * nteams + team;
    const bool active = L < nlines;
    C* line = base + (active ? L : 0) * ld;
    C a[16];
    if (active) {
      const auto ld0 = first(L);
#pragma unroll
      for (int q = 0; q < 16; ++q) a[q] = ld0(k + 16 * q);
      dft16<SIGN>(a);
    }
    __syncwarp();
    if (active) {
#pragma unroll
      for (int s = 0; s < 16; ++s) line[sidx(16 * s + k)] = a[s];
    }
    __syncwarp();
    if (active) {
      a[0] = line[sidx(16 * k)];
#pragma unroll
      for (int q = 1; q < 16; ++q) a[q] = ctw<SIGN>(line[sidx(16 * k + q)], w[16 * q]);
      dft16<SIGN>(a);
    }
    __syncwarp();
    if (active) {
#pragma unroll
      for (int s = 0; s < 16; ++s) line[sidx(k + 16 * s)] = a[s];
    }
    __syncwarp();
  }
}

// The same for FP64 lines in fixed point: 16 of the line's doubles become
// integers in each thread once the team has agreed on the line's scale, and
// the second stage hands its results to the line's out.
template <int SIGN, typename First, typename Out>
__device__ __forceinline__ void fft256_lines(double2* base, int ld, int nlines, const fxw* __restrict__ tw,
                                             const FftPlan& pl, First first, Out outs) {
  const int team = threadIdx.x >> 4;
  const int k = threadIdx.x & 15;
  const int nteams = blockDim.x >> 4;
  const int rounds = (nlines + nteams - 1) / nteams;
  const fxw* w = tw + pl.tw16_off + k;  // w[16 q] = w_256^{k q}
  for (int r = 0; r < rounds; ++r) {
    const int L = r * nteams + team;
    const bool active = L < nlines;
    double2* line = base + (active ? L : 0) * ld;
    fxc* fl = reinterpret_cast<fxc*>(line);
    fxc a[16];
    FxScale sc;
    const auto ld0 = first(active ? L : 0);
    const auto out = outs(active ? L : 0);
    if constexpr (LoadsInts<std::decay_t<decltype(ld0)>>::value) {
      sc = ld0.scale();
      if (active) {
#pragma unroll
        for (int q = 0; q < 16; ++q) a[q] = ld0(k + 16 * q);
      }
    } else {
      double2 v[16];
#pragma unroll
      for (int q = 0; q < 16; ++q) v[q] = make_double2(0.0, 0.0);
      if (active) {
#pragma unroll
        for (int q = 0; q < 16; ++q) v[q] = ld0(k + 16 * q);
      }
      sc = fx_begin<16, decltype(outs(0))::kNorm>(v, a, 16, 16.f);
    }
    dft16<SIGN>(a);
    __syncwarp();
    if (active) {
#pragma unroll
      for (int s = 0; s < 16; ++s) fl[sidx(16 * s + k)] = a[s];
    }
    __syncwarp();
    if (active) {
      a[0] = fl[sidx(16 * k)];
#pragma unroll
      for (int q = 1; q < 16; ++q) a[q] = ctw<SIGN>(fl[sidx(16 * k + q)], w[16 * q]);
      dft16<SIGN>(a);
    }
    __syncwarp();
    if (active) {
#pragma unroll
      for (int s = 0; s < 16; ++s) out(k + 16 * s, a[s], sc);
    }
    __syncwarp();
  }
}

// Lengths with a compile-time path: all 2^a 3^b 5^c from 8 to 256, and 512.
// (Below 16 points for the FP64 form: a line's scale and conversions at run-time
// radices made a step of 8^3 slower than FP64 arithmetic had, 168 against 141
// us; compiled 92.)
__host__ __device__ constexpr bool ct_length(int n) {
  if (n != 512 && (n < 8 || n > 256)) return false;
  while (n % 2 == 0) n /= 2;
  while (n % 3 == 0) n /= 3;
  while (n % 5 == 0) n /= 5;
  return n == 1;
}
// Radices of a compile-time length and the threads of its team.
struct CtPlan {
  int nst, r[4], tw;
};
// Lines that `threads` threads transform at once: teams of tw <= 32 threads
// fill a warp without crossing it, wider ones are whole warps.
__host__ __device__ constexpr int ct_teams(int tw, int threads) {
  return tw <= 32 ? (threads / 32) * (32 / tw) : threads / tw;
}
// Instructions of one butterfly of radix p in fixed point, its loads and
// stores included, to weigh the splits of a length against each other
// (counted, not measured: a complex sum 4, a product by a constant 11, a
// rotation 34).
__host__ __device__ constexpr int ct_cost(int p, bool first) {
  const int dft = p == 2 ? 8 : p == 3 ? 56 : p == 4 ? 32 : p == 5 ? 150 : p == 6 ? 136 : p == 8 ? 140 : p == 9 ? 472 :
                  p == 10 ? 340 : p == 12 ? 320 : p == 15 ? 730 : 490;
  return dft + 10 * p + (first ? 30 * p : 34 * (p - 1));
}
// The cheapest split into two or three radices for any team of 4 to 32
// threads (8 from n = 48) that hold at most 10 values each: instructions a
// line, times the share of a warp that its team takes; within 2 % the larger
// radices first (128: 8 x 8 x 2 before 8 x 4 x 4, FP32 stage 0.142 against
// 0.156 ms, FP64 0.513 against 0.503).  Fewer, larger radices
// in fewer threads (16 x 8 in 8 threads for n = 128) execute fewer instructions
// but leave too few loads in flight: FP32 x pass at 128^3 0.061 against
// 0.049 ms for 8 x 8 x 2 in 16.  256 and 512 keep the splits of their own paths.
__host__ __device__ constexpr CtPlan ct_plan(int n) {
  if (n == 256) return CtPlan{3, {8, 8, 4, 1}, 32};
  if (n == 512) return CtPlan{3, {8, 8, 8, 1}, 64};
  constexpr int R[11] = {2, 3, 4, 5, 6, 8, 9, 10, 12, 15, 16};
  CtPlan best{0, {1, 1, 1, 1}, 0};
  long cost = 0;
  for (int i = 10; i >= 0; --i)
    for (int j = 10; j >= 0; --j) {
      if (n % (R[i] * R[j])) continue;
      const int c = n / (R[i] * R[j]);
      bool known = c == 1;
      for (int k = 0; k < 11; ++k) known = known || c == R[k];
      if (!known) continue;
      const int r[3] = {R[i], R[j], c};
      const int nst = c == 1 ? 2 : 3;
      for (int tw = n < 48 ? 4 : 8; tw <= 32; ++tw) {
        long per = 0;
        bool ok = true;
        for (int s = 0; s < nst; ++s) {
          const int it = (n / r[s] + tw - 1) / tw;
          if (it * r[s] > 10) ok = false;
          per += (long)it * ct_cost(r[s], s == 0);
        }
        if (!ok) continue;
        const long line = per * 10000 / (32 / tw);
        if (best.nst == 0 || line * 50 < cost * 49) {
          cost = line;
          best = CtPlan{nst, {r[0], r[1], r[2], 1}, tw};
        }
      }
    }
  return best;
}
// Twiddles of the compile-time stages (the first has none).
__host__ __device__ constexpr int ct_tw_off(int n, int s) {
  const CtPlan p = ct_plan(n);
  int off = n == 256 ? 256 + 7 : 0, l = 1;  // (256: behind the 16 x 16 table, the run-time table's stages)
  for (int i = 0; i < s; ++i) {
    if (i > 0) off += l * (p.r[i] - 1);
    l *= p.r[i];
  }
  return off;
}
// Twiddles that a kernel compiled for PATH loads: the 16 x 16 table alone (at
// the start of the table) for the register path, the length's own stages'
// otherwise, all of them for run-time stages.
template <int PATH> __device__ __forceinline__ int tw_load(const FftPlan& pl) {
  return PATH == 256 ? pl.tw_total : pl.tw_pass;
}

// Stage S of compile-time length N: radix, sub-transform length, what is
// left, place in the twiddle table.
template <int N, int S> struct CtStage {
  static constexpr CtPlan kPlan = ct_plan(N);
  static constexpr int len(int s) { return s == 0 ? 1 : len(s - 1) * kPlan.r[s - 1]; }
  static constexpr int P = kPlan.r[S], L = len(S), M = N / (L * P), OFF = ct_tw_off(N, S), TW = kPlan.tw, NB = N / P;
  static constexpr int ITER = (NB + TW - 1) / TW;  // butterflies of a thread
  static constexpr bool FULL = NB % TW == 0;       // every thread has ITER of them
  static constexpr bool LAST = S + 1 == kPlan.nst;
};
// sidx(f M P + k + M q) for k < M as sidx at q = 0 plus a constant where the
// pads between 16 elements fall alike for every f and k
template <int M, int P> struct CtIndex {
  static constexpr bool kFold = (16 % M == 0 || M % 16 == 0) && (16 % (M * P) == 0 || (M * P) % 16 == 0);
  __device__ static __forceinline__ int at(int f, int k, int q) {
    if (kFold) return sidx(f * M * P + k) + (M * q + ((M * q) >> 4));
    return sidx(f * M * P + k + M * q);
  }
};

// a team's barrier: the warp's where teams do not cross warps
template <int TW> __device__ __forceinline__ void ct_sync() {
  if constexpr (TW <= 32) __syncwarp();
  else team_sync(TW);
}
// One stage of a compile-time length: everything but the thread's place is a
// constant.  active: whether the team has a line.
template <int SIGN, int N, int S, typename C, typename Ld, typename Out>
__device__ __forceinline__ void ct_stage(C* line, const typename TwOf<C>::type* __restrict__ tw, int tl, bool active,
                                         Ld load, Out out, FxScale& sc) {
  using G = CtStage<N, S>;
  constexpr bool FX = std::is_same<C, double2>::value;
  using A = std::conditional_t<FX, fxc, C>;
  constexpr int P = G::P, M = G::M, TW = G::TW, ITER = G::ITER;
  A a[ITER][P];
  A* fl = reinterpret_cast<A*>(line);
  if constexpr (S == 0 && FX && !LoadsInts<Ld>::value) {
    double2 v[ITER][P];
#pragma unroll
    for (int i = 0; i < ITER; ++i)
#pragma unroll
      for (int q = 0; q < P; ++q) v[i][q] = make_double2(0.0, 0.0);
    if (active) {
#pragma unroll
      for (int i = 0; i < ITER; ++i) {
        const int b = tl + i * TW;
        if (G::FULL || b < G::NB) {
#pragma unroll
          for (int q = 0; q < P; ++q) v[i][q] = load(b + M * q);
        }
      }
    }
    sc = fx_begin<ITER * P, Out::kNorm>(&v[0][0], &a[0][0], TW, Out::kNorm ? sqrtf((float)N) : 0.f);
  } else if constexpr (S == 0) {
    if constexpr (FX) sc = load.scale();
    if (active) {
#pragma unroll
      for (int i = 0; i < ITER; ++i) {
        const int b = tl + i * TW;
        if (G::FULL || b < G::NB) {
#pragma unroll
          for (int q = 0; q < P; ++q) a[i][q] = load(b + M * q);
        }
      }
    }
  } else if (active) {
#pragma unroll
    for (int i = 0; i < ITER; ++i) {
      const int b = tl + i * TW;
      if (G::FULL || b < G::NB) {
        const int f = b / M, k = b - f * M;
        const auto* w = tw + G::OFF + f * (P - 1);
        a[i][0] = fl[CtIndex<M, P>::at(f, k, 0)];
#pragma unroll
        for (int q = 1; q < P; ++q) a[i][q] = ctw<SIGN>(fl[CtIndex<M, P>::at(f, k, q)], w[q - 1]);
      }
    }
  }
  ct_sync<TW>();
  if (active) {
#pragma unroll
    for (int i = 0; i < ITER; ++i) {
      const int b = tl + i * TW;
      if (G::FULL || b < G::NB) {
        dftp<P, SIGN>(a[i]);
        // outputs b + q N / P
#pragma unroll
        for (int q = 0; q < P; ++q) {
          if constexpr (FX && G::LAST) out(b + q * (N / P), a[i][q], sc);
          else fl[CtIndex<N / P, P>::at(0, b, q)] = a[i][q];
        }
      }
    }
  }
  ct_sync<TW>();
}
template <int SIGN, int N, int S, typename C, typename First, typename Out>
__device__ __forceinline__ void fft_ct_stages(C* line, const typename TwOf<C>::type* __restrict__ tw, int tl,
                                              bool active, First first, Out out, FxScale& sc) {
  if constexpr (S < ct_plan(N).nst) {
    if constexpr (S == 0) ct_stage<SIGN, N, S>(line, tw, tl, active, first, out, sc);
    else ct_stage<SIGN, N, S>(line, tw, tl, active, 0, out, sc);
    fft_ct_stages<SIGN, N, S + 1>(line, tw, tl, active, first, out, sc);
  }
}

// Transform `nlines` lines of a CTA's shared-memory tile.  Line L starts at
// base + L*ld; its first stage reads through the loader first(L) returns (a
// functor idx -> value).  Every thread of the CTA must call this with the
// same plan.  A length-1 transform is the identity: the inputs are only
// copied into place.  Lines transformed in fixed point (kIsFx) hand their
// results to out(L); the others leave them in the line.
template <int SIGN, int PATH = kFftAny, typename C, typename First, typename Out>
__device__ __forceinline__ void fft_lines_from(C* base, int ld, int nlines,
                                               const typename TwOf<C>::type* __restrict__ tw,
                                               const FftPlan& pl, First first, Out out) {
  if (pl.n == 1 || pl.nst == 0) {
    if constexpr (!LoadsInts<std::decay_t<decltype(first(0))>>::value)  // (x lines only: Nx >= 2)
      for (int L = threadIdx.x; L < nlines; L += blockDim.x) base[L * ld] = first(L)(0);
    return;
  }
  if (PATH == kFft256 || (PATH == kFftAny && pl.tw16_off >= 0)) {
    fft256_lines<SIGN>(base, ld, nlines, tw, pl, first, out);
    return;
  }
  if (PATH == kFft256) return;
  if constexpr (ct_length(PATH)) {
    constexpr int TW = ct_plan(PATH).tw, G = TW <= 32 ? 32 / TW : 1;
    // lanes behind a warp's last whole team follow along without a line
    const int lane = threadIdx.x & 31;
    const int sub = TW <= 32 ? lane / TW : 0;
    const int team = TW <= 32 ? (int)(threadIdx.x >> 5) * G + sub : (int)threadIdx.x / TW;
    const int tl = TW <= 32 ? lane - sub * TW : (int)threadIdx.x - team * TW;
    const int nteams = ct_teams(TW, blockDim.x);
    const int rounds = (nlines + nteams - 1) / nteams;
    for (int r = 0; r < rounds; ++r) {
      const int L = r * nteams + team;
      const bool active = (TW > 32 || sub < G) && L < nlines;
      const int Lc = active ? L : 0;
      FxScale sc;
      fft_ct_stages<SIGN, PATH, 0>(base + Lc * ld, tw, tl, active, first(Lc), out(Lc), sc);
    }
  } else {
    const int TW = pl.team;
    const int nteams = blockDim.x / TW;
    const int team = threadIdx.x / TW;
    const int tl = threadIdx.x - team * TW;
    const int rounds = (nlines + nteams - 1) / nteams;
    for (int r = 0; r < rounds; ++r) {
      const int L = r * nteams + team;
      const bool active = L < nlines;
      const int Lc = active ? L : 0;
      fft_line_from<SIGN>(base + Lc * ld, tw, pl, tl, active, first(Lc), out(Lc));
    }
  }
}

// As above with the results left in the lines in every form.
template <int SIGN, int PATH = kFftAny, typename C, typename First>
__device__ __forceinline__ void fft_lines_from(C* base, int ld, int nlines,
                                               const typename TwOf<C>::type* __restrict__ tw,
                                               const FftPlan& pl, First first) {
  if constexpr (std::is_same<C, double2>::value)
    fft_lines_from<SIGN, PATH>(base, ld, nlines, tw, pl, first, [&](int L) { return FxOutLine{base + L * ld}; });
  else
    fft_lines_from<SIGN, PATH>(base, ld, nlines, tw, pl, first, [](int) { return 0; });
}

// As fft_lines_from on lines already in place.
template <int SIGN, int PATH = kFftAny, typename C>
__device__ __forceinline__ void fft_lines(C* base, int ld, int nlines, const typename TwOf<C>::type* __restrict__ tw,
                                          const FftPlan& pl) {
  if (pl.n == 1) return;
  fft_lines_from<SIGN, PATH>(base, ld, nlines, tw, pl, [&](int L) { return LineLoad<C>{base + L * ld}; });
}

// Copy a plan from global memory into shared memory (call before a barrier).
__device__ __forceinline__ void load_plan(FftPlan* s_plan, const FftPlan* __restrict__ g_plan) {
  const int nw = (int)(sizeof(FftPlan) / sizeof(int));
  const int* src = reinterpret_cast<const int*>(g_plan);
  int* dst = reinterpret_cast<int*>(s_plan);
  for (int i = threadIdx.x; i < nw; i += blockDim.x) dst[i] = src[i];
}

}  // namespace samgpu
