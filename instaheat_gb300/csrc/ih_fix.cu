// ih_fix.cu -- the transforms of the plain FP64 form in 64-bit block fixed
// point (ih_fix.cuh): passes along x and y, the derivative round trips, the
// real z passes and the fused z pass of the RHS.  Data
// in memory stay FP64 in the layouts of the other engines (ih_fft.cu); each
// pass converts a pencil on its way in and out of registers.
#include <math.h>
#include <vector>
#include "ih_internal.cuh"
#include "ih_fftcore.cuh"
#include "ih_fix.cuh"
#include "ih_zrow.cuh"

namespace ih {

// ---------------------------------------------------------------------------
// Passes along x or y: L = R1 R2, the two-step structure of the FP64 engines:
// thread (b, n1) holds x[n1 + R1 n2] of column b, an R2-point DFT, the table
// twiddle, one exchange through shared memory, an R1-point DFT.  Tiles of 8
// columns are 128-byte lines.  At 256^3 (55 launches of a DOPRI853 step, 3 to
// 4 arrays each): 272 us a launch against 1298 us on the FP64 pipe, 3.0 TB/s;
// 128^3: 47 against 163 us.  Both conversions are on the integer pipe: on the
// FP64 pipe (1.9 clocks per complex value and SM) they bound the pass, 340 and
// 57 us (inputs alone on the integer pipe 295 / 51, outputs alone 271 / 49).
template <int L> struct FxFac;
template <> struct FxFac<8> { static constexpr int R1 = 4, R2 = 2; };
template <> struct FxFac<16> { static constexpr int R1 = 4, R2 = 4; };
template <> struct FxFac<32> { static constexpr int R1 = 8, R2 = 4; };
template <> struct FxFac<64> { static constexpr int R1 = 8, R2 = 8; };
template <> struct FxFac<128> { static constexpr int R1 = 16, R2 = 8; };
template <> struct FxFac<256> { static constexpr int R1 = 16, R2 = 16; };
template <> struct FxFac<512> { static constexpr int R1 = 16, R2 = 32; };
template <> struct FxFac<12> { static constexpr int R1 = 4, R2 = 3; };
template <> struct FxFac<18> { static constexpr int R1 = 6, R2 = 3; };
template <> struct FxFac<24> { static constexpr int R1 = 6, R2 = 4; };
template <> struct FxFac<36> { static constexpr int R1 = 6, R2 = 6; };
template <> struct FxFac<48> { static constexpr int R1 = 8, R2 = 6; };
template <> struct FxFac<72> { static constexpr int R1 = 12, R2 = 6; };
template <> struct FxFac<96> { static constexpr int R1 = 12, R2 = 8; };
template <> struct FxFac<144> { static constexpr int R1 = 12, R2 = 12; };
template <> struct FxFac<192> { static constexpr int R1 = 16, R2 = 12; };
template <> struct FxFac<288> { static constexpr int R1 = 12, R2 = 24; };
template <> struct FxFac<384> { static constexpr int R1 = 16, R2 = 24; };
template <int L> __host__ __device__ constexpr int fx_p() {  // log2 rounded up
  return 64 - clog2(2 * L - 1) < 59 ? 64 - clog2(2 * L - 1) : 59;
}
template <int L> __host__ __device__ constexpr int fx_maxr() {
  return FxFac<L>::R1 > FxFac<L>::R2 ? FxFac<L>::R1 : FxFac<L>::R2;
}
template <int L, int B> __host__ __device__ constexpr int fx_threads() {
  return (fx_maxr<L>() * B + 31) / 32 * 32;
}
// row of the exchange buffer [L][B]: with 64-byte rows (B = 4) the rows that
// a group of lanes touches together have one parity, so rows swap with their
// neighbour on alternate blocks (as xrow in ih_fft.cu); 128-byte rows need
// nothing
template <int L, int B> __device__ __forceinline__ int fx_row(int r) {
  if (B >= 8) return r;
  constexpr int a = clog2(FxFac<L>::R1), b = clog2(FxFac<L>::R2);
  const int f = (a == b) ? (r >> a) : ((r >> a) ^ (r >> b));
  return r ^ (f & 1);
}
// the largest word of each column of the CTA: lanes of a warp that share a
// column, then the warps through red[warps][B]; every thread of the CTA calls
template <int B, int NT>
__device__ __forceinline__ unsigned fx_col_max(unsigned m, unsigned *red, int tid) {
#pragma unroll
  for (int o = B; o < 32; o <<= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
  if constexpr (NT == 32) return m;
  const int lane = tid & 31;
  if (lane < B) red[(tid >> 5) * B + lane] = m;
  __syncthreads();
#pragma unroll
  for (int w = 0; w < NT / 32; ++w) m = max(m, red[w * B + (tid & (B - 1))]);
  return m;
}

template <int L, int B, int S>
__global__ void __launch_bounds__(fx_threads<L, B>(), fx_maxr<L>() <= 16 ? 512 / fx_threads<L, B>() : 1)
    k_fx_xy(double2 *data, long long astride, long long sj, long long so, int mz, FxTab tw) {
  constexpr int R1 = FxFac<L>::R1, R2 = FxFac<L>::R2, NT = fx_threads<L, B>();
  extern __shared__ __align__(16) unsigned char smraw[];
  fx2 *ex = reinterpret_cast<fx2 *>(smraw);  // [L][B]
  __shared__ unsigned red[NT / 32 * B];
  const int tid = threadIdx.x, b = tid & (B - 1), q = tid / B;
  const int z0 = blockIdx.x * B;
  const bool col = b < mz - z0;
  double2 *base = data + blockIdx.z * astride + (long long)blockIdx.y * so + z0 + b;
  double2 x[R2];
#pragma unroll
  for (int n2 = 0; n2 < R2; ++n2)
    x[n2] = (col && q < R1) ? base[(long long)(q + R1 * n2) * sj] : make_double2(0.0, 0.0);
  const unsigned m = fx_col_max<B, NT>(fx_max_in(x), red, tid);
  const FxScale sc = fx_scale(m, fx_p<L>());
  if (q < R1) {
    fx2 v[R2];
    fx_load<true>(x, sc, v);
    fx_dft<R2, S>(v);
#pragma unroll
    for (int k2 = 0; k2 < R2; ++k2)
      ex[fx_row<L, B>(q * R2 + k2) * B + b] =
          k2 == 0 ? fx_quarter(v[k2]) : fx_cmul<S>(v[k2], fx_tw(tw, q * k2));
  }
  __syncthreads();
  if (q < R2) {
    fx2 u[R1];
#pragma unroll
    for (int n1 = 0; n1 < R1; ++n1) u[n1] = ex[fx_row<L, B>(n1 * R2 + q) * B + b];
    fx_dft<R1, S>(u);
    if (col) {
#pragma unroll
      for (int k1 = 0; k1 < R1; ++k1)
        base[(long long)(q + R2 * k1) * sj] = fx_store<true>(u[k1], sc.out + 2, sc);
    }
  }
}

// ---------------------------------------------------------------------------
// Derivative round trips along x or y (see k_fft_xy_rt): d1 = IFFT(i k FFT(Z))
// / (L nz), d2 = IFFT(-k^2 FFT(Z)) / (L nz).  c1, c2: k / 2^e1 and -k^2 / 2^e2
// in Q62 (first derivative 0 on the Nyquist index).  ACC (the y round trip):
// the coefficient of d2 takes -kz^2 too (cz, at the scale of c2), so that d2
// is the y and z part of the laplacian, and the x part in out1 is added.
// At 256^3: 347 us a round trip against 1359 us on the FP64 pipe, 128^3 58 us
// against 178.  Inputs convert on the FP64 pipe, outputs (two per input) on the
// integer pipe: 375 us with both on the former, 388 on the latter.
// Between the transforms the spectrum is brought to 2 bits above the inverse
// transform's p (the coefficients take 2), so no precision is lost whatever
// its size.
template <int L, int B, bool ACC>
__global__ void __launch_bounds__(fx_threads<L, B>(), fx_maxr<L>() <= 16 ? 384 / fx_threads<L, B>() : 1) k_fx_rt(
    const double2 *__restrict__ in, double2 *__restrict__ out0, double2 *out1, long long sj,
    long long so, int mz, FxTab tw, const long long *__restrict__ c1,
    const long long *__restrict__ c2, const long long *__restrict__ cz, int e1, int e2) {
  constexpr int R1 = FxFac<L>::R1, R2 = FxFac<L>::R2, NT = fx_threads<L, B>();
  extern __shared__ __align__(16) unsigned char smraw[];
  fx2 *ex0 = reinterpret_cast<fx2 *>(smraw), *ex1 = ex0 + L * B;  // [L][B] each
  __shared__ unsigned red[2][NT / 32 * B];
  const int tid = threadIdx.x, b = tid & (B - 1), q = tid / B;
  const int z0 = blockIdx.x * B;
  const bool col = b < mz - z0;
  const long long off = (long long)blockIdx.y * so + z0 + b;
  double2 x[R2];
#pragma unroll
  for (int n2 = 0; n2 < R2; ++n2)
    x[n2] = (col && q < R1) ? in[off + (long long)(q + R1 * n2) * sj] : make_double2(0.0, 0.0);
  if (z0 == 0 && q < R1) {
    // kz = 0: both derivatives of a constant are 0, so a pencil's first value
    // is taken off before the conversion (phi is a large constant plus
    // fluctuations, whose derivatives the constant's rounding would swamp)
    const double2 x0 = b == 0 ? in[off] : make_double2(0.0, 0.0);
    if (fx_absbits(x0.x) < 0x7ff00000u && fx_absbits(x0.y) < 0x7ff00000u) {
#pragma unroll
      for (int n2 = 0; n2 < R2; ++n2) {
        x[n2].x -= x0.x;
        x[n2].y -= x0.y;
      }
    }
  }
  const unsigned m = fx_col_max<B, NT>(fx_max_in(x), red[0], tid);
  const FxScale sc = fx_scale(m, fx_p<L>());
  if (q < R1) {
    fx2 v[R2];
    fx_load<false>(x, sc, v);
    fx_dft<R2, -1>(v);
#pragma unroll
    for (int k2 = 0; k2 < R2; ++k2)
      ex0[fx_row<L, B>(q * R2 + k2) * B + b] =
          k2 == 0 ? fx_quarter(v[k2]) : fx_cmul<-1>(v[k2], fx_tw(tw, q * k2));
  }
  __syncthreads();
  fx2 u[R1];
  if (q < R2) {
#pragma unroll
    for (int n1 = 0; n1 < R1; ++n1) u[n1] = ex0[fx_row<L, B>(n1 * R2 + q) * B + b];
    fx_dft<R1, -1>(u);  // u[k1] = X[q + R2 k1]
    if (z0 + b + q == 0) u[0] = fx_mk(0, 0);  // the constant: both coefficients are 0
  } else {
#pragma unroll
    for (int n1 = 0; n1 < R1; ++n1) u[n1] = fx_mk(0, 0);
  }
  const unsigned mu = fx_col_max<B, NT>(fx_max_int(u), red[1], tid);
  __syncthreads();  // ex0 is rewritten below (also where fx_col_max has no barrier)
  const int room = fx_room(mu, fx_p<L>() + 2);
  const FxShift sh = fx_shift_of(room);
  // the spectrum waits in the thread's own slots of ex1 between the two
  // inverse transforms (in registers it would halve the resident CTAs)
  auto slot = [&](int k1) { return (k1 * R2 + q) * B + b; };
  fx2 w[R1];
  if (q < R2) {
#pragma unroll
    for (int k1 = 0; k1 < R1; ++k1) {
      const fx2 v = fx_shift(u[k1], sh);
      ex1[slot(k1)] = v;
      const long long c = __ldg(c1 + q + R2 * k1);
      const int ch = fx_hi(c), cl = (int)c;
      w[k1] = fx_mk(-fx_mul(v.y, ch, cl), fx_mul(v.x, ch, cl));  // i k X
    }
    fx_dft<R1, +1>(w);
#pragma unroll
    for (int n1 = 0; n1 < R1; ++n1)
      ex0[fx_row<L, B>(q * R1 + n1) * B + b] =
          n1 == 0 ? fx_quarter(w[n1]) : fx_cmul<+1>(w[n1], fx_tw(tw, n1 * q));
    const long long z2 = ACC ? __ldg(cz + min(z0 + b, mz - 1)) : 0;
#pragma unroll
    for (int k1 = 0; k1 < R1; ++k1) {
      const fx2 v = ex1[slot(k1)];
      const long long c = __ldg(c2 + q + R2 * k1) + z2;
      const int ch = fx_hi(c), cl = (int)c;
      w[k1] = fx_mk(fx_mul(v.x, ch, cl), fx_mul(v.y, ch, cl));  // -k^2 X
    }
    fx_dft<R1, +1>(w);
  }
  __syncthreads();  // every slot of ex1 is read
  if (q < R2) {
#pragma unroll
    for (int n1 = 0; n1 < R1; ++n1)
      ex1[fx_row<L, B>(q * R1 + n1) * B + b] =
          n1 == 0 ? fx_quarter(w[n1]) : fx_cmul<+1>(w[n1], fx_tw(tw, n1 * q));
  }
  __syncthreads();
  if (q < R1) {
    // forward twiddle, coefficient and inverse twiddle took 2 bits each
    const int e = sc.out + 6 - room;
#pragma unroll
    for (int o = 0; o < 2; ++o) {
      const fx2 *ex = o ? ex1 : ex0;
      fx2 v[R2];
#pragma unroll
      for (int k2 = 0; k2 < R2; ++k2) v[k2] = ex[fx_row<L, B>(k2 * R1 + q) * B + b];
      fx_dft<R2, +1>(v);
      double2 *dst = (o ? out1 : out0) + off;
      if (col) {
#pragma unroll
        for (int n2 = 0; n2 < R2; ++n2) {
          double2 *d = dst + (long long)(q + R1 * n2) * sj;
          double2 r = fx_store<true>(v[n2], e + (o ? e2 : e1), sc);
          if (ACC && o == 1) {
            const double2 a = *d;
            r.x += a.x;
            r.y += a.y;
          }
          *d = r;
        }
      }
    }
  }
}

// ---------------------------------------------------------------------------
// z passes, on the engine of ih_zrow.cuh.  At 256^3: r2c 144 us an array
// against 606 us, c2r of four arrays 449 against 2564 us (FP64 pipe, wide rows
// and a warp per row); both conversions on the integer pipe (on the FP64 pipe
// 195 and 625 us).
struct NumFx {
  using C = fx2;
  using Tab = FxTab;
  __device__ static __forceinline__ C mk(long long x, long long y) { return fx_mk(x, y); }
  __device__ static __forceinline__ C add(C a, C b) { return a + b; }
  __device__ static __forceinline__ C sub(C a, C b) { return a - b; }
  __device__ static __forceinline__ C quarter(C v) { return fx_quarter(v); }
  __device__ static __forceinline__ C half(C v) { return fx_mk((v.x + 1) >> 1, (v.y + 1) >> 1); }
  __device__ static __forceinline__ C half_quarter(C v) {
    return fx_mk((v.x + 4) >> 3, (v.y + 4) >> 3);
  }
  template <int S>
  __device__ static __forceinline__ C cmul(C v, Tab t, int i) {
    return fx_cmul<S>(v, fx_tw(t, i));
  }
  template <int R, int S>
  __device__ static __forceinline__ void dft(C (&v)[R]) { fx_dft<R, S>(v); }
  __device__ static __forceinline__ C shfl(C v, int src) {
    return fx_mk(__shfl_sync(0xffffffffu, v.x, src), __shfl_sync(0xffffffffu, v.y, src));
  }
};
template <int H> struct FxZG : ZRow<NumFx, H> {
  // c2r: the split's 1/4 and the transform's growth H sqrt 2; r2c: the split
  // adds two values and the last bit of growth
  static constexpr int lg = clog2(2 * H - 1);  // log2 H, rounded up
  static constexpr int pc = 64 - lg < 58 ? 64 - lg : 58;
  static constexpr int pr = 63 - lg < 58 ? 63 - lg : 58;
};
constexpr int kFxWarps = 4;

// Real rows -> half spectra.  The row's first value is taken off before the
// conversion and nz times it added to X_0: a field that is a large constant
// plus fluctuations (the plain form's phi) is then resolved to 2^-p of its
// fluctuations.
template <int H>
__global__ void __launch_bounds__(32 * kFxWarps) k_fx_zr2c(
    const double *__restrict__ in, long long istride, double2 *__restrict__ out,
    long long ostride, long long rows, FxTab twh, FxTab twz) {
  using G = FxZG<H>;
  constexpr int A = G::A, B = G::B, E = G::E;
  __shared__ fx2 xs[kFxWarps][G::G * G::X];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int t = lane & (B - 1), grp = lane / B, gbase = lane & ~(B - 1);
  const long long row = ((long long)blockIdx.x * kFxWarps + warp) * G::G + grp;
  const bool valid = row < rows;
  const double2 *src = reinterpret_cast<const double2 *>(in + blockIdx.y * istride) + row * H;
  double2 x[A];
#pragma unroll
  for (int q = 0; q < B; ++q) {
#pragma unroll
    for (int e = 0; e < E; ++e)
      x[E * q + e] = valid ? src[E * t + e + A * q] : make_double2(0.0, 0.0);
  }
  double x0 = __shfl_sync(0xffffffffu, x[0].x, gbase);
  // an Inf or NaN stays in the row that has it: it reaches the scale below
  if (fx_absbits(x0) >= 0x7ff00000u) x0 = 0.0;
#pragma unroll
  for (int i = 0; i < A; ++i) {
    x[i].x -= x0;
    x[i].y -= x0;
  }
  const FxScale sc = fx_scale(zrow_max<FxZG<H>::B>(fx_max_in(x)), G::pr);
  fx2 v[A];
  fx_load<true>(x, sc, v);
  zrow_forward<NumFx, H>(v, t, &xs[warp][grp * G::X], twh);
  fx2 xH;
  zrow_r2c_post<NumFx, H>(v, t, gbase, twz, xH);
  if (valid) {
    double2 *dst = out + blockIdx.y * ostride + row * (H + 1);
#pragma unroll
    for (int m = 0; m < A; ++m) {
      double2 r = fx_store<true>(v[m], sc.out + 4, sc);
      if (m == 0 && t == 0) r.x += 2 * H * x0;
      dst[t + B * m] = r;
    }
    if (t == 0) dst[H] = fx_store<true>(xH, sc.out + 4, sc);
  }
}

// fetch a half-spectrum row: x[m] = X_(t + B m), xH = X_H on lane 0
template <int H>
__device__ __forceinline__ void fx_z_fetch(const double2 *row, int t, bool valid,
                                           double2 (&x)[FxZG<H>::A], double2 &xH) {
#pragma unroll
  for (int m = 0; m < FxZG<H>::A; ++m)
    x[m] = valid ? row[t + FxZG<H>::B * m] : make_double2(0.0, 0.0);
  xH = (valid && t == 0) ? row[H] : make_double2(0.0, 0.0);
}
template <int H, bool BITS>
__device__ __forceinline__ FxScale fx_z_load(double2 (&x)[FxZG<H>::A], double2 xH,
                                             fx2 (&v)[FxZG<H>::A], fx2 &vH) {
  double2 h[1] = {xH};
  fx2 u[1];
  const FxScale sc =
      fx_scale(zrow_max<FxZG<H>::B>(max(fx_max_in(x), fx_max_in(h))), FxZG<H>::pc);
  fx_load<BITS>(x, sc, v);
  fx_load<BITS>(h, sc, u);
  vH = u[0];
  return sc;
}

// Half spectra -> real rows.  The real part of X_0 is the row's mean times
// nz: it is left out of the transform and added to the outputs, for the same
// reason as above.
template <int H>
__global__ void __launch_bounds__(32 * kFxWarps) k_fx_zc2r(
    const double2 *__restrict__ in, long long istride, double *__restrict__ out,
    long long ostride, long long rows, FxTab twh, FxTab twz) {
  using G = FxZG<H>;
  constexpr int A = G::A, B = G::B, E = G::E;
  __shared__ fx2 xs[kFxWarps][G::G * G::X];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int t = lane & (B - 1), grp = lane / B, gbase = lane & ~(B - 1);
  const long long row = ((long long)blockIdx.x * kFxWarps + warp) * G::G + grp;
  const bool valid = row < rows;
  double2 x[A], xH;
  fx_z_fetch<H>(in + blockIdx.y * istride + row * (H + 1), t, valid, x, xH);
  double x0 = __shfl_sync(0xffffffffu, x[0].x, gbase);
  if (fx_absbits(x0) >= 0x7ff00000u) x0 = 0.0;
  if (t == 0) x[0].x -= x0;
  fx2 v[A], vH;
  const FxScale sc = fx_z_load<H, true>(x, xH, v, vH);
  zrow_c2r_prep<NumFx, H>(v, vH, t, gbase, twz);
  zrow_inverse<NumFx, H>(v, t, &xs[warp][grp * G::X], twh);
  if (valid) {
    double2 *dst = reinterpret_cast<double2 *>(out + blockIdx.y * ostride) + row * H;
#pragma unroll
    for (int q = 0; q < B; ++q) {
#pragma unroll
      for (int e = 0; e < E; ++e) {
        double2 r = fx_store<true>(v[E * q + e], sc.out + 4, sc);
        r.x += x0;
        r.y += x0;
        dst[E * t + e + A * q] = r;
      }
    }
  }
}

// ---------------------------------------------------------------------------
// The fused last z pass of the RHS (see k_fft_z_rhs_fused, ih_fft.cu): c2r of
// the derivative spectra, the laplacian written out, |grad phi|^2, rho, p and
// their FP64 sums, the six products d_i phi d_j phi and their r2c.  d/dx,
// d/dy, d/dz stay integers with a shared exponent per row, brought to 2^62;
// products of two rows are the upper 64 bits and go into the forward transform
// without a conversion.  rho and p are FP64.
//
// It takes about 2500 instructions per complex point; what bounds it is latency,
// so the three integer rows are not kept on the chip (96 KB of shared memory per
// CTA at H = 128, 8 warps an SM issuing on a third of the cycles) but written
// where the spectra of S_xz, S_yz and S_zz come to lie, each element by the
// thread that reads it back and at last overwrites it: they stay in the L2 (58 MB
// in flight), and the CTAs per SM below fit the registers.  At 256^3 2.47 -> 1.53
// ms (5.90 on the FP64 pipe), 192^3 1.61 -> 0.86, 128^3 0.182 -> 0.170, 96^3
// 0.115 -> 0.102 ms.  CTAs tried: A = 24 2 / 3: 969 / 855 us; A = 16 3 / 4 / 5:
// 1704 / 1528 / 1606; A = 12 3 / 4 / 5: 102 / 108 / 115; A = 8 5 / 6 / 8: 170 /
// 185 / 170 (128^3), 61 / 64 / 74 (64^3).
template <int H> struct FxZSmem {
  fx2 xs[kFxWarps][FxZG<H>::G * FxZG<H>::X];
};
template <int H> constexpr int fx_z_ctas() {
  constexpr int A = FxZG<H>::A;
  return A == 24 || A == 12 ? 3 : A == 16 ? 4 : A == 8 ? 5 : 6;
}

template <int H, bool ZSRC>
__global__ void __launch_bounds__(32 * kFxWarps, fx_z_ctas<H>()) k_fx_z_rhs(
    const double2 *d4, long long dstride, const double *__restrict__ yfl, const double *ysc,
    double *lap, double *pout, double *rhoout, double2 *s6, long long sstride, int gw,
    double *partials, Geom g, FxTab twh, FxTab twz, const long long *__restrict__ ckz,
    int ekz, int lognz) {
  using G = FxZG<H>;
  constexpr int A = G::A, B = G::B, E = G::E;
  extern __shared__ __align__(16) unsigned char smraw[];
  FxZSmem<H> &sm = *reinterpret_cast<FxZSmem<H> *>(smraw);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int t = lane & (B - 1), grp = lane / B, gbase = lane & ~(B - 1);
  const long long rows = (long long)g.nx * g.ny;
  const long long row = ((long long)blockIdx.x * kFxWarps + warp) * G::G + grp;
  const bool valid = row < rows;
  fx2 *xch = &sm.xs[warp][grp * G::X];
  // the thread's own elements of the three integer rows
  auto grad = [&](int a) {
    return reinterpret_cast<fx2 *>(s6 + (a == 0 ? 2 : a + 3) * sstride + row * (H + 1)) + t;
  };
  int ex[3];       // exponents of the three derivative rows
  double post[3];  // their slow factors (1 but for extreme rows)
#pragma unroll 1
  for (int i = 0; i < 4; ++i) {
    const int a = i < 2 ? 3 - i : i - 2;  // the laplacian, d/dz, d/dx, d/dy
    double2 x[A], xH;
    fx2 v[A], vH;
    FxScale sc;
    int e;
    fx_z_fetch<H>(d4 + (ZSRC && a == 2 ? 4 : a) * dstride + row * (H + 1), t, valid, x, xH);
    if (ZSRC && a == 2) {  // i kz Z / nz: the constant drops out
      if (t == 0) x[0] = make_double2(0.0, 0.0);
      sc = fx_z_load<H, false>(x, xH, v, vH);
#pragma unroll
      for (int m = 0; m < A; ++m) {
        const long long c = __ldg(ckz + t + B * m);
        const int ch = fx_hi(c), cl = (int)c;
        v[m] = fx_mk(-fx_mul(v[m].y, ch, cl), fx_mul(v[m].x, ch, cl));
      }
      vH = fx_mk(0, 0);  // zero on the Nyquist index
      e = sc.out + 2 + ekz - lognz;
    } else {
      sc = fx_z_load<H, false>(x, xH, v, vH);
      e = sc.out;
    }
    zrow_c2r_prep<NumFx, H>(v, vH, t, gbase, twz);
    zrow_inverse<NumFx, H>(v, t, xch, twh);
    e += 4;
    if (a == 3) {
      if (valid) {
        double2 *dst = reinterpret_cast<double2 *>(lap) + row * H;
#pragma unroll
        for (int q = 0; q < B; ++q) {
#pragma unroll
          for (int j = 0; j < E; ++j) dst[E * t + j + A * q] = fx_store<true>(v[E * q + j], e, sc);
        }
      }
    } else {
      const int room = fx_room(zrow_max<FxZG<H>::B>(fx_max_int(v)), 62);
      const FxShift sh = fx_shift_of(room);
#pragma unroll
      for (int m = 0; m < A; ++m) v[m] = fx_shift(v[m], sh);
      e -= room;
      if (valid) {
        fx2 *gr = grad(a);
#pragma unroll
        for (int m = 0; m < A; ++m) gr[B * m] = v[m];
      }
      if (a == 0) { ex[0] = e; post[0] = sc.post; }
      if (a == 1) { ex[1] = e; post[1] = sc.post; }
      if (a == 2) { ex[2] = e; post[2] = sc.post; }
    }
  }

  // rho and p; |grad phi|^2 from the integer squares at the largest exponent
  const double a_sc = ysc[4];
  const double inv_a2 = 1.0 / (a_sc * a_sc);
  const double hm2 = 0.5 * (g.mass * g.mass), third = 1.0 / 3.0;
  const long long N = g.N;
  const bool slow = post[0] != 1.0 || post[1] != 1.0 || post[2] != 1.0;
  const int em = max(ex[0], max(ex[1], ex[2]));
  const int r0 = min(2 * (em - ex[0]), 63), r1 = min(2 * (em - ex[1]), 63),
            r2 = min(2 * (em - ex[2]), 63);
  const int eg = 2 * em + 64;
  double dr = 0.0, dp = 0.0;
  if (valid) {
    const double2 *yp = reinterpret_cast<const double2 *>(yfl) + row * H;
    const double2 *yd = yp + N / 2, *ys = yp + N;
    double2 *po = reinterpret_cast<double2 *>(pout) + row * H;
    double2 *ro = reinterpret_cast<double2 *>(rhoout) + row * H;
    auto grad2 = [&](long long gx, long long gy, long long gz) {
      if (slow) {  // extreme rows: in FP64
        const double fx = fx_out<true>(gx, ex[0]) * post[0], fy = fx_out<true>(gy, ex[1]) * post[1],
                     fz = fx_out<true>(gz, ex[2]) * post[2];
        return fx * fx + fy * fy + fz * fz;
      }
      return fx_out<true>((fx_mul(gx, gx) >> r0) + (fx_mul(gy, gy) >> r1) + (fx_mul(gz, gz) >> r2), eg);
    };
#pragma unroll
    for (int q = 0; q < B; ++q) {
#pragma unroll
      for (int j = 0; j < E; ++j) {
        const int i = E * q + j;
        const long long at = E * t + j + A * q;
        const double2 ph = yp[at], dph = yd[at], ps = ys[at];
        const fx2 gx = grad(0)[B * i], gy = grad(1)[B * i], gz = grad(2)[B * i];
        double rx, ry, px, py;
        auto point = [&](double grad, double f, double d, double s, double &rho, double &p) {
          const double h = 0.5 - s, d2 = d * d, gi = grad * inv_a2;
          const double u = fma(-h, gi, gi);  // (1/2 + psi) |grad phi|^2 / a^2
          const double V = hm2 * f * f;
          rho = fma(h, d2, V) + u;
          p = fma(-third, u, fma(h, d2, -V));
        };
        point(grad2(gx.x, gy.x, gz.x), ph.x, dph.x, ps.x, rx, px);
        point(grad2(gx.y, gy.y, gz.y), ph.y, dph.y, ps.y, ry, py);
        po[at] = make_double2(px, py);
        if (rhoout) ro[at] = make_double2(rx, ry);
        dr += rx + ry;
        dp += px + py;
      }
    }
  }
  rhs_partial<32 * kFxWarps>(dr, dp, partials);
  if (!gw) return;

  // the six products and their forward transforms
#pragma unroll 1
  for (int pr = 0; pr < 6; ++pr) {
    const int ia = pr < 3 ? 0 : (pr < 5 ? 1 : 2);
    const int ib = pr < 3 ? pr : (pr < 5 ? pr - 2 : 2);
    fx2 v[A];
    const fx2 *ga = grad(ia), *gb = grad(ib);
#pragma unroll
    for (int m = 0; m < A; ++m) {
      const fx2 a = valid ? ga[B * m] : fx_mk(0, 0), b = valid ? gb[B * m] : fx_mk(0, 0);
      v[m] = fx_mk(fx_mul(a.x, b.x), fx_mul(a.y, b.y));
    }
    const int ea = ia == 0 ? ex[0] : (ia == 1 ? ex[1] : ex[2]);
    const int eb = ib == 0 ? ex[0] : (ib == 1 ? ex[1] : ex[2]);
    const double pa = ia == 0 ? post[0] : (ia == 1 ? post[1] : post[2]);
    const double pb = ib == 0 ? post[0] : (ib == 1 ? post[1] : post[2]);
    const int room = fx_room(zrow_max<FxZG<H>::B>(fx_max_int(v)), G::pr);
    const FxShift sh = fx_shift_of(room);
#pragma unroll
    for (int m = 0; m < A; ++m) v[m] = fx_shift(v[m], sh);
    zrow_forward<NumFx, H>(v, t, xch, twh);
    fx2 xH;
    zrow_r2c_post<NumFx, H>(v, t, gbase, twz, xH);
    const int e = ea + eb + 64 - room + 4;
    if (valid) {
      double2 *dst = s6 + pr * sstride + row * (H + 1);
      FxScale so;
      so.slow = slow;
      so.post = pa * pb;
#pragma unroll
      for (int m = 0; m < A; ++m) dst[t + B * m] = fx_store<true>(v[m], e, so);
      if (t == 0) dst[H] = fx_store<true>(xH, e, so);
    }
  }
}

// ---------------------------------------------------------------------------
// host side
static FxTab fx_tab(const void *p, int n) {
  FxTab t;
  t.a = reinterpret_cast<const int4 *>(p);
  t.b = reinterpret_cast<const int2 *>(t.a + n);
  return t;
}

static void fx_split(long long v, int &h, int &l) {
  l = (int)(unsigned)(unsigned long long)v;
  h = (int)((v - l) >> 32);
}

// exp(-2 pi i k / L), k < L, as FxTab entries
static int fx_upload_twiddles(Ctx *c, void **dst, int L) {
  std::vector<int> host(6 * (size_t)L);
  int *a = host.data(), *b = host.data() + 4 * (size_t)L;
  const long double pi = 3.14159265358979323846264338327950288L;
  for (int k = 0; k < L; ++k) {
    // octant reduction: the angle is at most pi/4, so that cos and sin round
    // alike for angles that are images of each other
    const int k8 = 8 * k / L, r = 8 * k - k8 * L;  // angle = k8 pi/4 + r pi/(4 L)
    const int odd = k8 & 1;
    const long double ang = pi / 4 * (odd ? L - r : r) / L;
    long double cs = cosl(ang), sn = sinl(ang);
    const int q = (k8 + odd) / 2;  // quarter turns around which the rest is +- ang
    if (odd) sn = -sn;
    long double re, im;
    switch (q & 3) {
      case 0: re = cs; im = sn; break;
      case 1: re = -sn; im = cs; break;
      case 2: re = -cs; im = -sn; break;
      default: re = sn; im = -cs; break;
    }
    const long long C = llrintl(ldexpl(re, 62)), S = llrintl(ldexpl(-im, 62));
    fx_split(C, a[4 * k], a[4 * k + 1]);
    fx_split(S - C, a[4 * k + 2], a[4 * k + 3]);
    fx_split(S + C, b[2 * k], b[2 * k + 1]);
  }
  IH_CUDA(c, cudaMalloc(dst, sizeof(int) * host.size()));
  c->dev_bytes += sizeof(int) * host.size();
  IH_CUDA(c, cudaMemcpy(*dst, host.data(), sizeof(int) * host.size(), cudaMemcpyHostToDevice));
  return IH_OK;
}

// derivative coefficients of one axis: c1[k] = k_f / (odd 2^e1) (0 on Nyquist),
// c2[k] = -k_f^2 / (odd 2^e2) in Q62, k folded to [-L/2, L/2); odd: the odd part
// of the transforms' 1 / N factors, whose power of two goes into the exponents
static void fx_coefs(std::vector<long long> &t, int L, int count, double unit, double unit2, int e1,
                     int e2, int odd1, int odd2) {
  for (int k = 0; k < count; ++k) {
    const int f = k > L / 2 ? k - L : k;
    t.push_back(2 * k == L ? 0 : llrintl(ldexpl((long double)unit * f / odd1, 62 - e1)));
  }
  for (int k = 0; k < count; ++k) {
    const int f = k > L / 2 ? L - k : k;
    t.push_back(-llrintl(ldexpl((long double)unit2 * f * f / odd2, 62 - e2)));
  }
}
static int fx_odd(int n) {
  while (n % 2 == 0) n /= 2;
  return n;
}
static int fx_twos(int n) {
  int s = 0;
  for (; n % 2 == 0; n /= 2) ++s;
  return s;
}
static int fx_exp(double v) {  // 2^e > v
  int e;
  frexp(v, &e);
  return e;
}

int fix_tables(Ctx *c) {
  const Geom &g = c->g;
  if (c->mixed) return IH_OK;
  const bool px = pencil_length(g.nx), py = pencil_length(g.ny), pz = zrow_length(g.h);
  IH_TRY(fx_upload_twiddles(c, &c->fx_tw[0], g.nx));
  IH_TRY(fx_upload_twiddles(c, &c->fx_tw[1], g.ny));
  IH_TRY(fx_upload_twiddles(c, &c->fx_tw[2], g.h));
  IH_TRY(fx_upload_twiddles(c, &c->fx_tw[3], g.nz));
  const double qx = g.kx2 * (g.nx / 2) * (g.nx / 2), qy = g.ky2 * (g.ny / 2) * (g.ny / 2),
               qz = g.kz2 * (g.nz / 2) * (g.nz / 2);
  c->fx_e[0] = fx_exp(g.kxmax);
  c->fx_e[1] = fx_exp(qx);
  c->fx_e[2] = fx_exp(g.kymax);
  c->fx_e[3] = fx_exp(qy + qz);
  c->fx_e[4] = fx_exp(g.kzmax);
  for (int e : c->fx_e)  // a box whose k leave the exponent range of the passes
    if (e < -200 || e > 200) return IH_OK;
  std::vector<long long> t;
  const int oz = fx_odd(g.nz), ox = fx_odd(g.nx) * oz, oy = fx_odd(g.ny) * oz;
  fx_coefs(t, g.nx, g.nx, g.kxu, g.kx2, c->fx_e[0], c->fx_e[1], ox, ox);
  fx_coefs(t, g.ny, g.ny, g.kyu, g.ky2, c->fx_e[2], c->fx_e[3], oy, oy);
  fx_coefs(t, g.nz, g.mz, g.kzu, g.kz2, c->fx_e[4], c->fx_e[3], oz, oy);
  IH_CUDA(c, cudaMalloc(&c->fx_coef, sizeof(long long) * t.size()));
  c->dev_bytes += sizeof(long long) * t.size();
  IH_CUDA(c, cudaMemcpy(c->fx_coef, t.data(), sizeof(long long) * t.size(),
                        cudaMemcpyHostToDevice));
  c->fx_can = (px ? 1 : 0) | (py ? 2 : 0) | (px && py && pz ? 8 | 16 : 0) | (pz ? 64 : 0);
  c->fx_on = c->fx_can;
  return IH_OK;
}

template <typename F>
static int fx_dispatch(int L, F &&f) {
  switch (L) {
    case 8: return f.template run<8>();
    case 16: return f.template run<16>();
    case 32: return f.template run<32>();
    case 64: return f.template run<64>();
    case 128: return f.template run<128>();
    case 256: return f.template run<256>();
    case 512: return f.template run<512>();
    case 12: return f.template run<12>();
    case 18: return f.template run<18>();
    case 24: return f.template run<24>();
    case 36: return f.template run<36>();
    case 48: return f.template run<48>();
    case 72: return f.template run<72>();
    case 96: return f.template run<96>();
    case 144: return f.template run<144>();
    case 192: return f.template run<192>();
    case 288: return f.template run<288>();
    case 384: return f.template run<384>();
    default: return IH_ERR_ARG;
  }
}
constexpr int kFxB = 8;  // columns of a tile: 128-byte lines

struct FxXY {
  Ctx *c;
  double2 *data;
  long long stride;
  int count, axis, sign, cols;
  template <int L>
  int run() {
    const Geom &g = c->g;
    const long long sj = axis == 0 ? (long long)g.ny * g.mz : g.mz;
    const long long so = axis == 0 ? g.mz : (long long)g.ny * g.mz;
    const int outer = axis == 0 ? g.ny : g.nx, mz = cols ? cols : g.mz;
    const FxTab tw = fx_tab(c->fx_tw[axis], L);
    const size_t sm = sizeof(fx2) * L * kFxB;
    const dim3 grid((mz + kFxB - 1) / kFxB, outer, count);
    auto kf = sign < 0 ? k_fx_xy<L, kFxB, -1> : k_fx_xy<L, kFxB, +1>;
    want_smem(kf, sm);
    kf<<<grid, fx_threads<L, kFxB>(), sm, c->stream>>>(data, stride, sj, so, mz, tw);
    return IH_OK;
  }
};
int fix_xy(Ctx *c, void *data, long long stride, int count, int axis, int sign, int cols) {
  return fx_dispatch(axis == 0 ? c->g.nx : c->g.ny,
                     FxXY{c, (double2 *)data, stride, count, axis, sign, cols});
}

struct FxRT {
  Ctx *c;
  const double2 *z;
  double2 *d1, *d2;
  int axis;
  template <int L>
  int run() {
    constexpr int B = 4;  // two exchange buffers and two spectra in registers
    const Geom &g = c->g;
    const long long sj = axis == 0 ? (long long)g.ny * g.mz : g.mz;
    const long long so = axis == 0 ? g.mz : (long long)g.ny * g.mz;
    const int outer = axis == 0 ? g.ny : g.nx;
    const FxTab tw = fx_tab(c->fx_tw[axis], L);
    const long long *cx = (const long long *)c->fx_coef, *cy = cx + 2 * g.nx,
                    *cz = cy + 2 * g.ny;
    const long long *c1 = axis == 0 ? cx : cy;
    const int scale = fx_twos(L) + fx_twos(g.nz);  // 1 / (L nz), its powers of two
    const int e1 = c->fx_e[2 * axis] - scale, e2 = c->fx_e[2 * axis + 1] - scale;
    const size_t sm = sizeof(fx2) * L * B * 2;
    const dim3 grid((g.mz + B - 1) / B, outer);
    auto kf = axis == 1 ? k_fx_rt<L, B, true> : k_fx_rt<L, B, false>;
    want_smem(kf, sm);
    kf<<<grid, fx_threads<L, B>(), sm, c->stream>>>(z, d1, d2, sj, so, g.mz, tw, c1, c1 + L,
                                                    cz + g.mz, e1, e2);
    return IH_OK;
  }
};
int fix_roundtrip(Ctx *c, const void *z, void *d1, void *d2, int axis) {
  return fx_dispatch(axis == 0 ? c->g.nx : c->g.ny,
                     FxRT{c, (const double2 *)z, (double2 *)d1, (double2 *)d2, axis});
}

struct FxZPass {
  Ctx *c;
  const void *in;
  long long istride;
  void *out;
  long long ostride;
  int count;
  bool forward;
  template <int H>
  int run() {
    const Geom &g = c->g;
    const long long rows = (long long)g.nx * g.ny, per = kFxWarps * FxZG<H>::G;
    const dim3 grid((unsigned)((rows + per - 1) / per), count);
    const FxTab th = fx_tab(c->fx_tw[2], H), tz = fx_tab(c->fx_tw[3], 2 * H);
    if (forward)
      k_fx_zr2c<H><<<grid, 32 * kFxWarps, 0, c->stream>>>((const double *)in, istride,
                                                          (double2 *)out, ostride, rows, th, tz);
    else
      k_fx_zc2r<H><<<grid, 32 * kFxWarps, 0, c->stream>>>((const double2 *)in, istride,
                                                          (double *)out, ostride, rows, th, tz);
    return IH_OK;
  }
};
template <typename F>
static int fx_z_dispatch(int H, F &&f) {
  switch (H) {
    case 4: return f.template run<4>();
    case 8: return f.template run<8>();
    case 16: return f.template run<16>();
    case 32: return f.template run<32>();
    case 64: return f.template run<64>();
    case 128: return f.template run<128>();
    case 256: return f.template run<256>();
    case 6: return f.template run<6>();
    case 12: return f.template run<12>();
    case 24: return f.template run<24>();
    case 48: return f.template run<48>();
    case 96: return f.template run<96>();
    case 192: return f.template run<192>();
    default: return IH_ERR_ARG;
  }
}
int fix_z(Ctx *c, const void *in, long long istride, void *out, long long ostride, int count,
          bool forward) {
  return fx_z_dispatch(c->g.h, FxZPass{c, in, istride, out, ostride, count, forward});
}

struct FxZRhs {
  Ctx *c;
  const double2 *d4;
  const double *yfl, *ysc;
  double *lap, *p, *rho;
  double2 *s6;
  int gw;
  double *partials;
  int zsrc;
  template <int H>
  int run() {
    const Geom &g = c->g;
    const long long rows = (long long)g.nx * g.ny, per = kFxWarps * FxZG<H>::G;
    const unsigned nblk = (unsigned)((rows + per - 1) / per);
    if (2LL * nblk > c->partials_cap) {
      c->err = "grid too large for the RHS partial-sum buffer";
      return IH_ERR_ARG;
    }
    const FxTab th = fx_tab(c->fx_tw[2], H), tz = fx_tab(c->fx_tw[3], 2 * H);
    const long long *cz = (const long long *)c->fx_coef + 2 * g.nx + 2 * g.ny;
    auto kf = zsrc ? k_fx_z_rhs<H, true> : k_fx_z_rhs<H, false>;
    const size_t sm = sizeof(FxZSmem<H>);
    want_smem(kf, sm);
    c->z_blocks = (int)nblk;
    kf<<<nblk, 32 * kFxWarps, sm, c->stream>>>(d4, g.M, yfl, ysc, lap, p, rho, s6, g.M, gw,
                                               partials, g, th, tz, cz, c->fx_e[4],
                                               fx_twos(g.nz));
    return IH_OK;
  }
};
int fix_z_rhs(Ctx *c, const void *d4, const void *yfl, const double *ysc, void *lap, void *p,
              void *rho, void *s6, int gw, double *partials, int zsrc) {
  return fx_z_dispatch(c->g.h, FxZRhs{c, (const double2 *)d4, (const double *)yfl, ysc,
                                      (double *)lap, (double *)p, (double *)rho, (double2 *)s6,
                                      gw, partials, zsrc});
}

}  // namespace ih
