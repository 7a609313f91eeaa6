// ih_fixz.cu -- the z passes of the plain FP64 form in 64-bit block fixed point
// (ih_fix.cuh): r2c, c2r and the fused z pass of the RHS.
#include "ih_internal.cuh"
#include "ih_fftcore.cuh"
#include "ih_fix.cuh"
#include "ih_zrow.cuh"

namespace ih {

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
template <int H> struct FxZG : ZRow<NumFx, H> {};
// bits for a row's integers (fx_scale).  r2c: the split adds two outputs, each below
// sqrt(2) S / 4.  c2r: the split comes first and rotates the sum of two values, each
// in one thread's part
constexpr int kFxRealP = 62, kFxRealS = 63, kFxHalfP = 61, kFxHalfS = 64;
template <int B>
__device__ __forceinline__ FxSize fx_row_size(FxSize z) {
#pragma unroll
  for (int o = 1; o < B; o <<= 1) z = fx_join_lanes(z, o);
  return z;
}
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
  const FxScale sc = fx_scale(fx_row_size<B>(fx_size(x)), kFxRealP, kFxRealS);
  fx2 v[A];
  fx_load<true>(x, sc, v);
  zrow_forward<NumFx, H>(v, t, &xs[warp][grp * G::X], twh);
  fx2 xH;
  zrow_r2c_post<NumFx, H>(v, t, gbase, twz, xH);
  if (valid) {
    double2 *dst = out + blockIdx.y * ostride + row * (H + 1);
#pragma unroll
    for (int m = 0; m < A; ++m) {
      double2 r = fx_store(v[m], sc.out + 4, sc);
      if (m == 0 && t == 0) r.x += 2 * H * x0;
      dst[t + B * m] = r;
    }
    if (t == 0) dst[H] = fx_store(xH, sc.out + 4, sc);
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
  FxSize z = fx_size(x), zH = fx_size(h);
  zH.e -= zH.s == 0 ? kFxBad : 0;  // (zero on the other lanes: no part of the size)
  z = fx_join(z, zH);
  const FxScale sc = fx_scale(fx_row_size<FxZG<H>::B>(z), kFxHalfP, kFxHalfS);
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
        double2 r = fx_store(v[E * q + e], sc.out + 4, sc);
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
// without a conversion.  rho and p are FP64.  First the parts, then two kernels
// made of them.
struct FxZIn {
  const double2 *d4;  // d/dx, d/dy, (d/dz), laplacian, (Z) in (x, y, kz)
  long long dstride;
  const double *ckz;  // kz / nz
  int zsrc;  // d/dz from Z in slot 4
  FxTab twh, twz;
};
struct FxZLane {
  int t, gbase;
  bool valid;
  long long row;
  fx2 *xch;
};
// spectrum row a (3: the laplacian) -> integers at the exponent returned
template <int H>
__device__ __forceinline__ int fx_z_deriv(const FxZIn &in, int a, const FxZLane &ln,
                                          fx2 (&v)[FxZG<H>::A], FxScale &sc) {
  constexpr int A = FxZG<H>::A, B = FxZG<H>::B;
  double2 x[A], xH;
  fx2 vH;
  fx_z_fetch<H>(in.d4 + (in.zsrc && a == 2 ? 4 : a) * in.dstride + ln.row * (H + 1), ln.t, ln.valid,
                x, xH);
  if (in.zsrc && a == 2) {  // i kz Z / nz, in FP64: the row's size is that of the product
#pragma unroll
    for (int m = 0; m < A; ++m) {
      const double f = __ldg(in.ckz + ln.t + B * m);
      x[m] = make_double2(-x[m].y * f, x[m].x * f);
    }
    xH = make_double2(0.0, 0.0);  // zero on the Nyquist index
  }
  sc = fx_z_load<H, false>(x, xH, v, vH);
  zrow_c2r_prep<NumFx, H>(v, vH, ln.t, ln.gbase, in.twz);
  zrow_inverse<NumFx, H>(v, ln.t, ln.xch, in.twh);
  return sc.out + 4;
}
// bring a row to 2^bits; the exponent taken off
template <int H>
__device__ __forceinline__ int fx_z_norm(fx2 (&v)[FxZG<H>::A], int bits) {
  const int room = fx_room(zrow_max<FxZG<H>::B>(fx_max_int(v)), bits);
  const FxShift sh = fx_shift_of(room);
#pragma unroll
  for (int m = 0; m < FxZG<H>::A; ++m) v[m] = fx_shift(v[m], sh);
  return room;
}
template <int H>
__device__ __forceinline__ void fx_z_lap(const fx2 (&v)[FxZG<H>::A], int e, const FxScale &sc,
                                         const FxZLane &ln, double *lap) {
  constexpr int A = FxZG<H>::A, B = FxZG<H>::B, E = FxZG<H>::E;
  if (!ln.valid) return;
  double2 *dst = reinterpret_cast<double2 *>(lap) + ln.row * H;
#pragma unroll
  for (int q = 0; q < B; ++q) {
#pragma unroll
    for (int j = 0; j < E; ++j)
      dst[E * ln.t + j + A * q] = fx_store(v[E * q + j], e, sc);
  }
}
// the six products: xx, xy, xz, yy, yz, zz
__device__ __forceinline__ int fx_z_first(int pr) { return pr < 3 ? 0 : (pr < 5 ? 1 : 2); }
__device__ __forceinline__ int fx_z_second(int pr) { return pr < 3 ? pr : (pr < 5 ? pr - 2 : 2); }
// a product at exponent e (slow rows: times post) -> its half spectrum
template <int H>
__device__ __forceinline__ void fx_z_product(fx2 (&v)[FxZG<H>::A], int e, bool slow, double post,
                                             const FxZIn &in, const FxZLane &ln, double2 *spec) {
  constexpr int A = FxZG<H>::A, B = FxZG<H>::B;
  float p = fx_sum_int(v), s = p;
#pragma unroll
  for (int o = 1; o < B; o <<= 1) {
    p = fmaxf(p, __shfl_xor_sync(0xffffffffu, p, o));
    s = __fadd_ru(s, __shfl_xor_sync(0xffffffffu, s, o));
  }
  // (the sums themselves, without the sqrt(2): a bit more than kFxRealS)
  const int room = fx_room_sum(p, s, 38, 62, 64);
  const FxShift sh = fx_shift_of(room);
#pragma unroll
  for (int m = 0; m < A; ++m) v[m] = fx_shift(v[m], sh);
  e += 4 - room;
  zrow_forward<NumFx, H>(v, ln.t, ln.xch, in.twh);
  fx2 xH;
  zrow_r2c_post<NumFx, H>(v, ln.t, ln.gbase, in.twz, xH);
  if (!ln.valid) return;
  double2 *dst = spec + ln.row * (H + 1);
  FxScale so;
  so.slow = slow;
  so.post = post;
#pragma unroll
  for (int m = 0; m < A; ++m) dst[ln.t + B * m] = fx_store(v[m], e, so);
  if (ln.t == 0) dst[H] = fx_store(xH, e, so);
}
// rho and p of a point; |grad phi|^2 from the integer squares at the largest
// exponent of the three rows.  These resolve it to 2^-60 of the row's largest, which
// at 2^-13 of that and below is more than the FP64 engines' derivatives leave in a
// square: there from the derivatives as FP64 (a field that varies alike along
// all axes has one such point in 10^5; everywhere, 1.39 -> 1.53 ms at 256^3).
struct FxZPoint {
  double inv_a2, hm2;
  int ex[3];       // exponents of the three derivative rows
  double post[3];  // their slow factors (1 but for extreme rows)
  bool slow;
  int r[3], eg;
  __device__ __forceinline__ void init(double a, double mass) {
    inv_a2 = 1.0 / (a * a);
    hm2 = 0.5 * (mass * mass);
    slow = post[0] != 1.0 || post[1] != 1.0 || post[2] != 1.0;
    const int em = max(ex[0], max(ex[1], ex[2]));
#pragma unroll
    for (int i = 0; i < 3; ++i) r[i] = min(2 * (em - ex[i]), 63);
    eg = 2 * em + 64;
  }
  __device__ __forceinline__ double grad2(long long gx, long long gy, long long gz) const {
    const long long s = (fx_mul_sum(gx, gx) >> r[0]) + (fx_mul_sum(gy, gy) >> r[1]) +
                        (fx_mul_sum(gz, gz) >> r[2]);
    if (slow || s < 1LL << 47) {  // extreme rows, small gradients
      const double fx = fx_out_bits(gx, ex[0]) * post[0], fy = fx_out_bits(gy, ex[1]) * post[1],
                   fz = fx_out_bits(gz, ex[2]) * post[2];
      return fx * fx + fy * fy + fz * fz;
    }
    return fx_out_bits(s, eg);
  }
  __device__ __forceinline__ void operator()(double grad, double f, double d, double s, double &rho,
                                             double &p) const {
    const double h = 0.5 - s, d2 = d * d, gi = grad * inv_a2;
    const double u = fma(-h, gi, gi);  // (1/2 + psi) |grad phi|^2 / a^2
    const double V = hm2 * f * f;
    rho = fma(h, d2, V) + u;
    p = fma(-(1.0 / 3.0), u, fma(h, d2, -V));
  }
};
struct FxZOut {
  const double *yfl;
  double *p, *rho;
  long long N;
  // register i of a lane: elements 2 at, 2 at + 1 of the row
  template <int H>
  __device__ __forceinline__ void point(const FxZPoint &pt, const FxZLane &ln, int i, fx2 gx,
                                        fx2 gy, fx2 gz, double &dr, double &dp) const {
    constexpr int A = FxZG<H>::A, E = FxZG<H>::E;
    const long long at = ln.row * H + E * ln.t + i % E + A * (i / E);
    const double2 *y = reinterpret_cast<const double2 *>(yfl) + at;
    const double2 ph = y[0], dph = y[N / 2], ps = y[N];
    double rx, ry, px, py;
    pt(pt.grad2(gx.x, gy.x, gz.x), ph.x, dph.x, ps.x, rx, px);
    pt(pt.grad2(gx.y, gy.y, gz.y), ph.y, dph.y, ps.y, ry, py);
    reinterpret_cast<double2 *>(p)[at] = make_double2(px, py);
    if (rho) reinterpret_cast<double2 *>(rho)[at] = make_double2(rx, ry);
    dr += rx + ry;
    dp += px + py;
  }
};

// A warp per group of rows, one transform after the other, for grids that fill
// the GPU.
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
// 185 / 170 (128^3).  The points two at a time in a loop instead of unrolled: 1.58 ->
// 1.39 ms at 256^3, 895 -> 827 us at 192^3, 172 -> 169 at 128^3 (the unrolled kernel
// waited for instructions).
template <int H> constexpr int fx_z_ctas() {
  constexpr int A = FxZG<H>::A;
  return A == 24 || A == 12 ? 3 : A == 16 ? 4 : A == 8 ? 5 : 6;
}
template <int H>
__global__ void __launch_bounds__(32 * kFxWarps, fx_z_ctas<H>()) k_fx_z_rhs(
    const FxZIn in, const FxZOut out, const double *ysc, double *lap, double2 *s6,
    long long sstride, int gw, double *partials, long long rows, double mass) {
  using G = FxZG<H>;
  constexpr int A = G::A, B = G::B;
  __shared__ fx2 xs[kFxWarps][G::G * G::X];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, grp = lane / B;
  FxZLane ln;
  ln.t = lane & (B - 1);
  ln.gbase = lane & ~(B - 1);
  ln.row = ((long long)blockIdx.x * kFxWarps + warp) * G::G + grp;
  ln.valid = ln.row < rows;
  ln.xch = &xs[warp][grp * G::X];
  // the thread's own elements of the three integer rows
  auto grad = [&](int a) {
    return reinterpret_cast<fx2 *>(s6 + (a == 0 ? 2 : a + 3) * sstride + ln.row * (H + 1)) + ln.t;
  };
  FxZPoint pt;
#pragma unroll 1
  for (int i = 0; i < 4; ++i) {
    // the laplacian, d/dz, d/dx, d/dy: the integers of dx and dy may take the
    // place of a source of d/dz
    const int a = i < 2 ? 3 - i : i - 2;
    fx2 v[A];
    FxScale sc;
    int e = fx_z_deriv<H>(in, a, ln, v, sc);
    if (a == 3) {
      fx_z_lap<H>(v, e, sc, ln, lap);
    } else {
      e -= fx_z_norm<H>(v, 62);
      if (ln.valid) {
        fx2 *gr = grad(a);
#pragma unroll
        for (int m = 0; m < A; ++m) gr[B * m] = v[m];
      }
      if (a == 0) { pt.ex[0] = e; pt.post[0] = sc.post; }
      if (a == 1) { pt.ex[1] = e; pt.post[1] = sc.post; }
      if (a == 2) { pt.ex[2] = e; pt.post[2] = sc.post; }
    }
  }
  pt.init(ysc[4], mass);
  double dr = 0.0, dp = 0.0;
  if (ln.valid) {
#pragma unroll 2
    for (int i = 0; i < A; ++i)  // (unrolled, the kernel waits for instructions)
      out.point<H>(pt, ln, i, grad(0)[B * i], grad(1)[B * i], grad(2)[B * i], dr, dp);
  }
  rhs_partial<32 * kFxWarps>(dr, dp, partials);
  if (!gw) return;
#pragma unroll 1
  for (int pr = 0; pr < 6; ++pr) {
    const int ia = fx_z_first(pr), ib = fx_z_second(pr);
    fx2 v[A];
    const fx2 *ga = grad(ia), *gb = grad(ib);
#pragma unroll
    for (int m = 0; m < A; ++m) {
      const fx2 a = ln.valid ? ga[B * m] : fx_mk(0, 0), b = ln.valid ? gb[B * m] : fx_mk(0, 0);
      v[m] = fx_mk(fx_mul_sum(a.x, b.x), fx_mul_sum(a.y, b.y));
    }
    const int ea = ia == 0 ? pt.ex[0] : (ia == 1 ? pt.ex[1] : pt.ex[2]);
    const int eb = ib == 0 ? pt.ex[0] : (ib == 1 ? pt.ex[1] : pt.ex[2]);
    const double pa = ia == 0 ? pt.post[0] : (ia == 1 ? pt.post[1] : pt.post[2]);
    const double pb = ib == 0 ? pt.post[0] : (ib == 1 ? pt.post[1] : pt.post[2]);
    fx_z_product<H>(v, ea + eb + 64, pt.slow, pa * pb, in, ln, s6 + pr * sstride);
  }
}

// Eight warps per group of rows, for grids with few rows: four transform the
// derivatives, then six the products and two take half the points each, so
// that the chain is two transforms long instead of ten: the pass then has to do
// with one transform's latency, not with its throughput.  One warp a group / eight,
// by groups of rows: 128 (32^3) 28.9 / 12.4 us, 144 (48^3) 74 / 22.7, 384
// (96x64x48) 94 / 53, 512 (64^3) 62 / 41, 1024 (128x64x64) 72 / 58, 1152 (96^3)
// 105 / 100, 2048 (128x128x64, 128x128x32) 97 / 96 and 53 / 58.  CTAs of A = 8
// per SM 2 / 3: 38.8 / 41.2 (64^3), 63 / 58 us (128x64x64).
template <int H> struct FxZCo {
  fx2 xs[6][FxZG<H>::G * FxZG<H>::X];
  fx2 grad[3][FxZG<H>::A][32];
  int ex[3][FxZG<H>::G];
  double post[3][FxZG<H>::G];
};
// (nx >= ny >= nz: rows longer than 96 come in larger numbers)
template <int H> constexpr bool kFxZCo = H <= 48;
template <int H> constexpr int fx_zco_ctas() {
  return FxZG<H>::A == 12 ? 2 : 3;
}
template <int H>
__global__ void __launch_bounds__(256, fx_zco_ctas<H>()) k_fx_z_rhs_co(
    const FxZIn in, const FxZOut out, const double *ysc, double *lap, double2 *s6,
    long long sstride, int gw, double *partials, long long rows, double mass) {
  using G = FxZG<H>;
  constexpr int A = G::A, B = G::B;
  extern __shared__ __align__(16) unsigned char smraw[];
  FxZCo<H> &sm = *reinterpret_cast<FxZCo<H> *>(smraw);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, grp = lane / B;
  FxZLane ln;
  ln.t = lane & (B - 1);
  ln.gbase = lane & ~(B - 1);
  ln.row = (long long)blockIdx.x * G::G + grp;
  ln.valid = ln.row < rows;
  ln.xch = &sm.xs[warp < 6 ? warp : 0][grp * G::X];
  if (warp < 4) {
    fx2 v[A];
    FxScale sc;
    int e = fx_z_deriv<H>(in, warp, ln, v, sc);
    if (warp == 3) {
      fx_z_lap<H>(v, e, sc, ln, lap);
    } else {
      e -= fx_z_norm<H>(v, 62);
#pragma unroll
      for (int m = 0; m < A; ++m) sm.grad[warp][m][lane] = v[m];
      if (ln.t == 0) {
        sm.ex[warp][grp] = e;
        sm.post[warp][grp] = sc.post;
      }
    }
  }
  __syncthreads();
  double dr = 0.0, dp = 0.0;
  if (warp >= 6) {
    FxZPoint pt;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
      pt.ex[a] = sm.ex[a][grp];
      pt.post[a] = sm.post[a][grp];
    }
    pt.init(ysc[4], mass);
    if (ln.valid) {
#pragma unroll
      for (int j = 0; j < A / 2; ++j) {
        const int i = j + (warp - 6) * (A / 2);
        out.point<H>(pt, ln, i, sm.grad[0][i][lane], sm.grad[1][i][lane], sm.grad[2][i][lane], dr,
                     dp);
      }
    }
  } else if (gw) {
    const int ia = fx_z_first(warp), ib = fx_z_second(warp);
    fx2 v[A];
#pragma unroll
    for (int m = 0; m < A; ++m) {
      const fx2 a = sm.grad[ia][m][lane], b = sm.grad[ib][m][lane];
      v[m] = fx_mk(fx_mul_sum(a.x, b.x), fx_mul_sum(a.y, b.y));
    }
    const bool slow =
        sm.post[0][grp] != 1.0 || sm.post[1][grp] != 1.0 || sm.post[2][grp] != 1.0;
    fx_z_product<H>(v, sm.ex[ia][grp] + sm.ex[ib][grp] + 64, slow,
                    sm.post[ia][grp] * sm.post[ib][grp], in, ln, s6 + warp * sstride);
  }
  rhs_partial<256>(dr, dp, partials);
}

// ---------------------------------------------------------------------------
// host side
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
    const long long rows = (long long)g.nx * g.ny, groups = (rows + FxZG<H>::G - 1) / FxZG<H>::G;
    const bool co = kFxZCo<H> && groups <= 8LL * c->num_sms;  // see k_fx_z_rhs_co
    const unsigned nblk = (unsigned)(co ? groups : (groups + kFxWarps - 1) / kFxWarps);
    if (2LL * nblk > c->partials_cap) {
      c->err = "grid too large for the RHS partial-sum buffer";
      return IH_ERR_ARG;
    }
    const double *kz = (const double *)c->fx_coef + 2 * g.nx + 2 * g.ny;
    const FxZIn in{d4, g.M, kz, zsrc, fx_tab(c->fx_tw[2], H), fx_tab(c->fx_tw[3], 2 * H)};
    const FxZOut out{yfl, p, rho, g.N};
    c->z_blocks = (int)nblk;
    if constexpr (kFxZCo<H>) {
      if (co) {
        want_smem(k_fx_z_rhs_co<H>, sizeof(FxZCo<H>));
        k_fx_z_rhs_co<H><<<nblk, 256, sizeof(FxZCo<H>), c->stream>>>(
            in, out, ysc, lap, s6, g.M, gw, partials, rows, g.mass);
        return IH_OK;
      }
    }
    k_fx_z_rhs<H><<<nblk, 32 * kFxWarps, 0, c->stream>>>(in, out, ysc, lap, s6, g.M, gw, partials,
                                                         rows, g.mass);
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
