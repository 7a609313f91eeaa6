// ih_fix.cuh -- 64-bit block fixed point for the transforms of the plain FP64
// form.
//
// An FP64 addition issues at 1.8 per clock per SM on this GPU (measured:
// independent DADD chains, 152 SMs at 1.92 GHz; DFMA 2.1), a 64-bit integer
// addition at 60, and the product of two 64-bit fractions (the upper 64 bits,
// one IMAD.WIDE and two IMAD.HI) at 7.5 against 1.8 DMUL.  A transform is
// mostly additions, so the passes here hold a pencil as 64-bit integers that
// share one exponent, the butterflies are integer additions (exact), and every
// multiplication by a twiddle rounds to a unit.  The exponent follows from the
// pencil's sum of magnitudes (FxSize), which bounds every value on the way,
// whatever the pencil holds: white noise has its units where the largest
// value's worst growth would put them, a pencil with one dominant value 2^-57 of
// that value.  Errors of a pass (2-norm) are 0.2 to 0.7 of those in FP64 for
// white noise, a spike, a falling or a single-wave spectrum of 8 to 512 points.
//
// Growth: sqrt(2) S bounds the sum of the magnitudes.  The part of it that one
// thread holds bounds its first DFT, whose outputs are rotated (x + y: a factor
// sqrt(2)), so that part's S stays below 2^62; the multiplication by a table twiddle
// keeps the upper 64 bits of a product with a Q62 fraction, a factor 1/4, so that
// the second DFT is bounded by sqrt(2) S / 4, its inner rotations by S / 2, and S
// may be 2^64.
#pragma once
#include "ih_internal.cuh"
#include "ih_fftcore.cuh"

namespace ih {

struct __align__(16) fx2 {
  long long x, y;
};

// a table twiddle c + i s as the three products of a complex multiplication
// need it: c, c - s, c + s in Q62, each split as high * 2^32 + low with a
// signed low word (a = {c high, c low, c-s high, c-s low}, b = {c+s})
struct FxTab {
  const int4 *a;
  const int2 *b;
};
struct FxW {
  int4 a;
  int2 b;
};
__device__ __forceinline__ FxW fx_tw(const FxTab &t, int i) {
  FxW w;
  w.a = __ldg(t.a + i);
  w.b = __ldg(t.b + i);
  return w;
}

__device__ __forceinline__ fx2 fx_mk(long long x, long long y) {
  fx2 r;
  r.x = x;
  r.y = y;
  return r;
}
__device__ __forceinline__ fx2 operator+(fx2 a, fx2 b) { return fx_mk(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ fx2 operator-(fx2 a, fx2 b) { return fx_mk(a.x - b.x, a.y - b.y); }

// high * 2^32 + low with a signed low word
__device__ __forceinline__ int fx_hi(long long a) {
  return (int)(a >> 32) + (int)((unsigned)a >> 31);
}
// a w / 2^64 from the split halves of both, the low * low product (a quarter of a
// unit at most, of either sign) left out.  A product with zero is zero in the first two
// forms, so that what cancels exactly in FP64 transforms cancels here.
//   fx_mul_low: both cross products round down, by a unit on average together, half
//   a unit for a small a; for differences of two products, where that goes away.
__device__ __forceinline__ long long fx_mul_low(int ah, int al, int wh, int wl) {
  return (long long)ah * wh + (__mulhi(ah, wl) + __mulhi(al, wh));
}
//   fx_mul: al w rounds to nearest, so a small a has no bias, a large one half a
//   unit.  (Both to nearest: 5% more time in every pass that has it.)
__device__ __forceinline__ long long fx_mul(int ah, int al, int wh, int wl) {
  const int c = __mulhi(ah, wl) + (int)(((long long)al * wh + 0x80000000LL) >> 32);
  return (long long)ah * wh + c;
}
//   fx_mul_sum: the + 1 returns the average unit; one unit for a zero.  For sums
//   of a few products, where a unit is nothing.
__device__ __forceinline__ long long fx_mul_sum(int ah, int al, int wh, int wl) {
  const int c = __mulhi(ah, wl) + __mulhi(al, wh) + 1;
  return (long long)ah * wh + c;
}
__device__ __forceinline__ long long fx_mul(long long a, int wh, int wl) {
  return fx_mul(fx_hi(a), (int)a, wh, wl);
}
// by a 64-bit constant or variable fraction
__device__ __forceinline__ long long fx_mul(long long a, long long w) {
  return fx_mul(fx_hi(a), (int)a, fx_hi(w), (int)w);
}
__device__ __forceinline__ long long fx_mul_sum(long long a, long long w) {
  return fx_mul_sum(fx_hi(a), (int)a, fx_hi(w), (int)w);
}
// v (c + i s) / 4 (S = -1) or v (c - i s) / 4 (S = +1), the table holding the
// forward twiddle; each component the difference of two products
template <int S>
__device__ __forceinline__ fx2 fx_cmul(fx2 v, const FxW &w) {
  const long long m = v.x + v.y;
  const long long k = fx_mul_low(fx_hi(m), (int)m, w.a.x, w.a.y);
  const int xh = fx_hi(v.x), xl = (int)v.x, yh = fx_hi(v.y), yl = (int)v.y;
  if (S < 0)
    return fx_mk(k - fx_mul_low(yh, yl, w.b.x, w.b.y), k - fx_mul_low(xh, xl, w.a.z, w.a.w));
  return fx_mk(k - fx_mul_low(yh, yl, w.a.z, w.a.w), k - fx_mul_low(xh, xl, w.b.x, w.b.y));
}
// v / 4, the trivial twiddle
__device__ __forceinline__ fx2 fx_quarter(fx2 v) { return fx_mk((v.x + 2) >> 2, (v.y + 2) >> 2); }

// rotation by D x 90 degrees
template <int D>
__device__ __forceinline__ fx2 fx_rot90(fx2 v) {
  if ((D & 3) == 0) return v;
  if ((D & 3) == 1) return fx_mk(-v.y, v.x);
  if ((D & 3) == 2) return fx_mk(-v.x, -v.y);
  return fx_mk(v.y, -v.x);
}
// v exp(2 pi i M / 32) at v's own scale: quarter turns and a rotation by at
// most 45 degrees, which is three shears (tan, sin, tan of Q64 fractions
// below 1/2) or, at 45 degrees, a sum and a difference by sqrt(1/2) = 1 -
// 0.29289...
constexpr long long kFxOneMinusSqrtHalf = 0x4afb0ccc06219b7cLL;  // 1 - sqrt(1/2)
constexpr long long kFxTanPi16 = 0x32ebebc0aa62b00fLL;           // tan(pi/16)
constexpr long long kFxSinPi8 = 0x61f78a9abaa58b47LL;            // sin(pi/8)
constexpr long long kFxTanPi32 = 0x1936bb8c5b2da262LL;           // tan(pi/32)
constexpr long long kFxSinPi16 = 0x31f17078d34c156dLL;           // sin(pi/16)
constexpr long long kFxTan3Pi32 = 0x4da820d5718f6f14LL;          // tan(3 pi/32)
constexpr long long kFxOneMinusSin3Pi16 = 0x71c626328cb9bc9bLL;  // 1 - sin(3 pi/16)

template <int M>
__device__ __forceinline__ fx2 fx_rot32(fx2 v) {
  constexpr int m = ((M % 32) + 32) % 32;
  constexpr int q = (m + 4) / 8;  // quarter turns; the rest r in (-45, 45]
  constexpr int r = m - 8 * q;    // -4 .. 3 units of 11.25 degrees
  v = fx_rot90<q>(v);
  if (r == 0) return v;
  if (r == -4) {  // 45 degrees clockwise: (x + y, y - x) sqrt(1/2)
    const long long a = v.x + v.y, b = v.y - v.x;
    return fx_mk(a - fx_mul(a, kFxOneMinusSqrtHalf), b - fx_mul(b, kFxOneMinusSqrtHalf));
  }
  constexpr int ra = r < 0 ? -r : r;
  constexpr long long T = ra == 1 ? kFxTanPi32 : ra == 2 ? kFxTanPi16 : kFxTan3Pi32;
  if (r > 0) {
    v.x -= fx_mul(v.y, T);
    if (ra == 3)
      v.y += v.x - fx_mul(v.x, kFxOneMinusSin3Pi16);
    else
      v.y += fx_mul(v.x, ra == 1 ? kFxSinPi16 : kFxSinPi8);
    v.x += fx_mul(v.y, -T);  // (of the sign that the first product's bias does not have)
  } else {
    v.x += fx_mul(v.y, T);
    if (ra == 3)
      v.y -= v.x - fx_mul(v.x, kFxOneMinusSin3Pi16);
    else
      v.y -= fx_mul(v.x, ra == 1 ? kFxSinPi16 : kFxSinPi8);
    v.x -= fx_mul(v.y, -T);
  }
  return v;
}

// a[j][k] <- a[j][k] exp(S 2 pi i j k / R)
template <int R, int S, int J, int M, int I>
__device__ __forceinline__ void fx_twist(fx2 (&a)[J][M]) {
  if constexpr (I < J * M) {
    constexpr int j = I / M, k = I % M;
    if constexpr (j > 0 && k > 0) a[j][k] = fx_rot32<S * j * k * (32 / R)>(a[j][k]);
    fx_twist<R, S, J, M, I + 1>(a);
  }
}
// in-register DFT of R <= 32 points (a power of two, or three times one), v[k]
// <- sum_n v[n] exp(S 2 pi i nk/R)
constexpr long long kFxOneMinusSqrt34 = 0x224c28bd3d9aac62LL;  // 1 - sqrt(3)/2
template <int R, int S>
__device__ __forceinline__ void fx_dft(fx2 (&v)[R]) {
  if constexpr (R % 3 == 0) {
    // Good and Thomas' index maps n = Q n1 + 3 n2, k = (k mod 3, k mod Q) leave no
    // twiddles between the factors 3 and Q
    constexpr int Q = R / 3;
    fx2 a[3][Q];
#pragma unroll
    for (int n = 0; n < Q; ++n) {
      const fx2 x0 = v[(3 * n) % R], x1 = v[(Q + 3 * n) % R], x2 = v[(2 * Q + 3 * n) % R];
      const fx2 s = x1 + x2, d = x1 - x2;
      const fx2 m = fx_mk(x0.x - ((s.x + 1) >> 1), x0.y - ((s.y + 1) >> 1));
      const fx2 h = fx_rot90<S>(fx_mk(d.x - fx_mul(d.x, kFxOneMinusSqrt34),
                                      d.y - fx_mul(d.y, kFxOneMinusSqrt34)));
      a[0][n] = x0 + s;
      a[1][n] = m + h;
      a[2][n] = m - h;
    }
#pragma unroll
    for (int k = 0; k < 3; ++k) fx_dft<Q, S>(a[k]);
#pragma unroll
    for (int k = 0; k < R; ++k) v[k] = a[k % 3][k % Q];
  } else if constexpr (R == 2) {
    const fx2 a = v[0], b = v[1];
    v[0] = a + b;
    v[1] = a - b;
  } else if constexpr (R == 4) {
    const fx2 s02 = v[0] + v[2], d02 = v[0] - v[2], s13 = v[1] + v[3];
    const fx2 j13 = fx_rot90<S>(v[1] - v[3]);
    v[0] = s02 + s13;
    v[2] = s02 - s13;
    v[1] = d02 + j13;
    v[3] = d02 - j13;
  } else if constexpr (R > 1) {  // one twiddle per value, as in reg_dft
    constexpr int J = R == 8 ? 2 : 4, M = R / J;
    fx2 a[J][M];
#pragma unroll
    for (int j = 0; j < J; ++j) {
#pragma unroll
      for (int m = 0; m < M; ++m) a[j][m] = v[j + J * m];
      fx_dft<M, S>(a[j]);
    }
    fx_twist<R, S, J, M, 0>(a);
#pragma unroll
    for (int k = 0; k < M; ++k) {
      fx2 b[J];
#pragma unroll
      for (int j = 0; j < J; ++j) b[j] = a[j][k];
      fx_dft<J, S>(b);
#pragma unroll
      for (int q = 0; q < J; ++q) v[k + M * q] = b[q];
    }
  }
}

// ---------------------------------------------------------------------------
// FP64 <-> fixed point of one pencil
__device__ __forceinline__ unsigned fx_absbits(double a) {
  return (unsigned)__double2hiint(a) & 0x7fffffffu;
}
// Size of a pencil, an upper bound of its sum of magnitudes over sqrt(2): what one
// thread holds is below 2^(e - 1022), the pencil at most s 2^(e - 1042); s = 0 if
// every value is 0, e = kFxBad if one is an Inf or NaN.  Groups of up to four values
// count with their largest component (each value by itself would cost a tenth of a
// pass in time and hardly change the bound).
constexpr int kFxBad = 4096;
struct FxSize {
  int e;
  unsigned s;
};
template <int R>
__device__ __forceinline__ FxSize fx_size(const double2 (&x)[R]) {
  constexpr int G = R % 4 == 0 ? 4 : (R % 3 == 0 ? 3 : R), NG = R / G;
  unsigned m[NG], all = 0, low = 0;
#pragma unroll
  for (int g = 0; g < NG; ++g) {
    m[g] = 0;
#pragma unroll
    for (int i = g; i < R; i += NG) {
      m[g] = max(m[g], max(fx_absbits(x[i].x), fx_absbits(x[i].y)));
      low |= (unsigned)(__double2loint(x[i].x) | __double2loint(x[i].y));
    }
    all = max(all, m[g]);
  }
  // a component is below (upper bits of its mantissa + 1) 2^(exponent - 1043)
  const unsigned E = all >> 20;
  unsigned s = NG;
#pragma unroll
  for (int g = 0; g < NG; ++g)
    s += __funnelshift_rc((m[g] & 0xfffffu) | 0x100000u, 0u, E - (m[g] >> 20));
  s *= G;
  const int n = 32 - __clz((int)s);  // 2^20 < s < 2^n
  FxSize z;
  z.e = E == 2047 ? kFxBad : (int)E + n - 21;
  z.s = (all | low) ? (s >> (n - 20)) + 1 : 0;
  return z;
}
__device__ __forceinline__ FxSize fx_join(FxSize a, FxSize b) {
  auto up = [](unsigned s, int d) { return (s + ((1u << d) - 1)) >> d; };
  FxSize z;
  z.e = max(a.e, b.e);
  z.s = up(a.s, min(z.e - a.e, 31)) + up(b.s, min(z.e - b.e, 31));
  return z;
}
__device__ __forceinline__ FxSize fx_join_lanes(FxSize z, int o) {
  FxSize b;
  b.e = __shfl_xor_sync(0xffffffffu, z.e, o);
  b.s = __shfl_xor_sync(0xffffffffu, z.s, o);
  return fx_join(z, b);
}
struct FxScale {
  int in;       // exponent added to the inputs: integer = round(x 2^in)
  int out;      // exponent of the result so far: value = integer 2^out
  bool slow;    // the pencil needs the factors below
  double pre, post;
};
// The integers of a pencil of size z: a thread's below 2^bp in all, the pencil's
// below 2^bs.
// The common case (e for values of 2^-323 to 2^37) takes exponents for which
// adding `in` to the exponent field of any component (zeros and subnormals
// included) stays a finite number, and for which the exponents of products of
// two pencils stay in range; other pencils are brought there by an exact power
// of two, and a pencil with an Inf or NaN comes out as NaN.
__device__ __forceinline__ FxScale fx_scale(FxSize z, int bp, int bs) {
  FxScale s;
  int E = z.e;
  const int bits = min(bp, bs - (12 - __clz((int)z.s)));  // z.s < 2^(32 - clz)
  s.slow = E < 700 || E > 1060;
  s.pre = s.post = 1.0;
  if (s.slow) {
    int d;  // exponent taken off: values of the order of one, or as near as a factor comes
    if (E == kFxBad) {
      d = 0;
      E = 1023;
    } else {
      d = E < 1 ? -1000 : (E > 2023 ? 1000 : E - 1023);
      E = (E < 1 ? 1 : E) - d;
    }
    s.pre = __hiloint2double((1023 - d) << 20, 0);
    s.post = __hiloint2double((1023 + d) << 20, 0);
    if (z.e == kFxBad) {
      s.pre = 0.0;
      s.post = __longlong_as_double(0x7ff8000000000000LL);
    }
    if (z.s == 0) s.post = 0.0;  // all zero
  }
  s.in = bits + 1022 - E;
  s.out = -s.in;
  return s;
}
// Conversion on the FP64 pipe (2.1 per clock and SM) ...
__device__ __forceinline__ long long fx_in_pipe(double a, const FxScale &s) {
  return __double2ll_rn(
      __hiloint2double(__double2hiint(a) + s.in * (1 << 20), __double2loint(a)));
}
// ... and on the integer pipe (about 3.5 per clock and SM): the mantissa, its
// leading one put in, shifted to the pencil's exponent, and back by a count of
// leading zeros; both round to nearest
__device__ __forceinline__ long long fx_in_shift(double a, int r) {
  const unsigned hi = (unsigned)__double2hiint(a), lo = (unsigned)__double2loint(a);
  // a = m 2^(e - 1075) with m < 2^53; m 2^10 is below 2^63 and goes right by
  // r > 0 bits, one of them in the rounding
  unsigned long long m = ((unsigned long long)((hi & 0xfffffu) | 0x100000u) << 32 | lo) << 10;
  // (shr clamps: a count of 64 or more, as for zeros, gives 0)
  asm("shr.u64 %0, %0, %1;" : "+l"(m) : "r"(r));
  const long long t = (long long)((m + 1) >> 1);
  return (int)hi < 0 ? -t : t;
}
__device__ __forceinline__ long long fx_in_bits(double a, const FxScale &s) {
  return fx_in_shift(a, 1084 - s.in - (int)(((unsigned)__double2hiint(a) >> 20) & 0x7ff));
}
__device__ __forceinline__ double fx_out_bits(long long v, int e) {
  const unsigned long long u = (unsigned long long)(v < 0 ? -v : v);
  const int lz = __clzll((long long)u);
  const unsigned long long n = u << (lz & 63);
  const unsigned long long m = (n >> 11) + ((n >> 10) & 1);  // 2^52 .. 2^53
  const int h = (int)(m >> 32) + (1085 - lz + e) * (1 << 20);
  return __hiloint2double(u == 0 ? 0 : (h | ((int)(v >> 32) & (int)0x80000000)), (int)(unsigned)m);
}
template <bool BITS>
__device__ __forceinline__ long long fx_in(double a, const FxScale &s) {
  return BITS ? fx_in_bits(a, s) : fx_in_pipe(a, s);
}
template <bool BITS, int R>
__device__ __forceinline__ void fx_load(double2 (&x)[R], const FxScale &s, fx2 (&v)[R]) {
  if (s.slow) {
#pragma unroll
    for (int i = 0; i < R; ++i) {
      x[i].x = s.pre == 0.0 ? 0.0 : x[i].x * s.pre;
      x[i].y = s.pre == 0.0 ? 0.0 : x[i].y * s.pre;
    }
  }
#pragma unroll
  for (int i = 0; i < R; ++i) v[i] = fx_mk(fx_in<BITS>(x[i].x, s), fx_in<BITS>(x[i].y, s));
}
// value of v at exponent e, through the slow factor where the pencil has one
__device__ __forceinline__ double2 fx_store(fx2 v, int e, const FxScale &s) {
  double2 r = make_double2(fx_out_bits(v.x, e), fx_out_bits(v.y, e));
  if (s.slow) {
    r.x *= s.post;
    r.y *= s.post;
  }
  return r;
}
// |high word| of integers, and the shift that brings a largest such word just
// below 2^bits (a left shift loses nothing; a right shift rounds)
__device__ __forceinline__ unsigned fx_abshi(long long a) {
  const int h = (int)(a >> 32);
  return (unsigned)(h ^ (h >> 31));
}
template <int R>
__device__ __forceinline__ unsigned fx_max_int(const fx2 (&v)[R]) {
  unsigned m = 0;
#pragma unroll
  for (int i = 0; i < R; ++i) m = max(m, max(fx_abshi(v[i].x), fx_abshi(v[i].y)));
  return m;
}
__device__ __forceinline__ int fx_room(unsigned maxhi, int bits) {
  return bits - (64 - __clz(maxhi));  // |v| < 2^(64 - clz(maxhi))
}
// The same for integers: the sum of |Re| + |Im| over what a thread holds, in
// units of 2^38, rounded up; and the shift that makes room for a transform, from the
// largest such sum p and all of them together s (units of 2^unit)
template <int R>
__device__ __forceinline__ float fx_sum_int(const fx2 (&v)[R]) {
  unsigned s = R;
#pragma unroll
  for (int i = 0; i < R; ++i) s += (fx_abshi(v[i].x) + fx_abshi(v[i].y)) >> 6;
  return __uint2float_ru(s);
}
__device__ __forceinline__ int fx_float_exp(float f) {  // f < 2^(this), f > 0
  return (__float_as_int(f) >> 23) - 126;
}
__device__ __forceinline__ int fx_room_sum(float p, float s, int unit, int bp, int bs) {
  return min(bp - fx_float_exp(p), bs - fx_float_exp(s)) - unit;
}
struct FxShift {
  int l, r;
  long long half;
};
__device__ __forceinline__ FxShift fx_shift_of(int s) {
  FxShift f;
  f.l = max(s, 0);
  f.r = max(-s, 0);
  f.half = (1LL << f.r) >> 1;
  return f;
}
__device__ __forceinline__ long long fx_shift(long long v, const FxShift &f) {
  return ((v << f.l) + f.half) >> f.r;
}
__device__ __forceinline__ fx2 fx_shift(fx2 v, const FxShift &f) {
  return fx_mk(fx_shift(v.x, f), fx_shift(v.y, f));
}

// ---------------------------------------------------------------------------
// Sums sum_j c_j x_j of a few FP64 numbers per element, off the FP64 pipe:
// c_j = C_j 2^(k_j - 62) with |C_j| <= 2^62, the x_j 2^(k_j) as integers at the
// exponent of the largest of them (2^61), the upper halves of the products added
// up.  With n <= 15 terms the sum stays below 2^63, and its error is at most a
// unit per term, 2^-57 of the largest product: below that of an FP64 sum, whose
// terms each round to 2^-53 of a partial sum.
constexpr int kFxSum = 3;  // terms from which FP64 sums of vectors are summed so
__device__ __forceinline__ long long fx_mul_sum(int ah, int al, FxCoef c) {
  return fx_mul_sum(ah, al, c.h, c.l);
}
__device__ __forceinline__ int fx_exponent(double x, int k) {  // biased, of x 2^k
  return ((__double2hiint(x) >> 20) & 0x7ff) + k;
}
// the mantissa of x with its leading one and sign, 2^61 to 2^62 (a zero's or
// subnormal's is of no use), split for products: x = m 2^(fx_exponent - 1084)
struct FxMantissa {
  int h, l;
};
__device__ __forceinline__ FxMantissa fx_mantissa(double x) {
  const int hi = __double2hiint(x);
  long long v = ((long long)((hi & 0xfffff) | 0x100000) << 32 | (unsigned)__double2loint(x)) << 9;
  if (hi < 0) v = -v;
  FxMantissa m;
  m.h = fx_hi(v);
  m.l = (int)v;
  return m;
}
struct FxPoint {
  bool fast;  // every x_j finite, the sums' exponents in range (k_j within 64)
  int in;     // integer = x_j 2^(k_j + in)
  __device__ __forceinline__ explicit FxPoint(int E) {  // the largest fx_exponent
    fast = E >= 200 && E <= 1900;
    in = 61 + 1022 - E;
  }
  __device__ __forceinline__ long long get(double x, int e) const {
    return fx_in_shift(x, 1084 - in - e);
  }
  // (k: of coefficients that share one exponent, which get() then leaves out)
  __device__ __forceinline__ double put(long long v, int k = 0) const {
    return fx_out_bits(v, 2 + k - in);
  }
};

// host side: a twiddle table of n entries, and the power of two in n
inline FxTab fx_tab(const void *p, int n) {
  FxTab t;
  t.a = reinterpret_cast<const int4 *>(p);
  t.b = reinterpret_cast<const int2 *>(t.a + n);
  return t;
}

inline int fx_twos(int n) {
  int s = 0;
  for (; n % 2 == 0; n /= 2) ++s;
  return s;
}
inline void fx_split(long long v, int &h, int &l) {
  l = (int)(unsigned)(unsigned long long)v;
  h = (int)((v - l) >> 32);
}
// the exponent of a coefficient, kFxNone for one that FxPoint does not take
// (zero, or outside 2^-64 .. 2^64); c as a fraction of 2^k
constexpr int kFxNone = 1 << 20;
inline int fx_coef_exp(double c) {
  int e = 0;
  const double m = frexp(c, &e);
  return fabs(m) >= 0.5 && fabs(m) < 1.0 && e >= -64 && e <= 64 ? e : kFxNone;
}
inline FxCoef fx_coef(double c, int k) {
  FxCoef f;
  fx_split(llrint(ldexp(c, 62 - k)), f.h, f.l);
  f.k = k;
  return f;
}

}  // namespace ih
