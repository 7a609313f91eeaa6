// ih_fix.cu -- the transforms of the plain FP64 form in 64-bit block fixed
// point (ih_fix.cuh): passes along x and y, the derivative round trips and the
// tables (the z passes: ih_fixz.cu).  Data
// in memory stay FP64 in the layouts of the other engines (ih_fft.cu); each
// pass converts a pencil on its way in and out of registers.
#include <math.h>
#include <string.h>
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
// 6 arrays each): 501 us a launch on average, 3.0 TB/s (six arrays 556 us; on the
// FP64 pipe four took 1298 us); 128^3: 82 us.  Sizing a pencil by its sum of
// magnitudes takes 6% of that (473 and 75 us by its largest value).  Both
// conversions are on the integer pipe: on the FP64 pipe (1.9 clocks per complex
// value and SM) they bounded the pass, 340 against 272 us of four arrays (inputs
// alone on the integer pipe 295, outputs alone 271).
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
// over each column of the CTA: lanes of a warp that share a column, then the warps
// through red[warps][B]; every thread of the CTA calls
template <int B, int NT>
__device__ __forceinline__ FxSize fx_col_size(FxSize z, FxSize *red, int tid) {
#pragma unroll
  for (int o = B; o < 32; o <<= 1) z = fx_join_lanes(z, o);
  if constexpr (NT == 32) return z;
  const int lane = tid & 31;
  if (lane < B) red[(tid >> 5) * B + lane] = z;
  __syncthreads();
  z = red[tid & (B - 1)];
#pragma unroll
  for (int w = 1; w < NT / 32; ++w) z = fx_join(z, red[w * B + (tid & (B - 1))]);
  return z;
}
// the largest sum of a thread and the sum of all (fx_room_sum), of two pencils
template <int B, int NT>
__device__ __forceinline__ void fx_col_sums(float2 &p, float2 &s, float4 *red, int tid) {
  auto join = [&](float4 o) {
    p.x = fmaxf(p.x, o.x);
    p.y = fmaxf(p.y, o.y);
    s.x = __fadd_ru(s.x, o.z);
    s.y = __fadd_ru(s.y, o.w);
  };
#pragma unroll
  for (int o = B; o < 32; o <<= 1) {
    float4 b;
    b.x = __shfl_xor_sync(0xffffffffu, p.x, o);
    b.y = __shfl_xor_sync(0xffffffffu, p.y, o);
    b.z = __shfl_xor_sync(0xffffffffu, s.x, o);
    b.w = __shfl_xor_sync(0xffffffffu, s.y, o);
    join(b);
  }
  if constexpr (NT == 32) return;
  const int lane = tid & 31;
  if (lane < B) red[(tid >> 5) * B + lane] = make_float4(p.x, p.y, s.x, s.y);
  __syncthreads();
  p = s = make_float2(0.0f, 0.0f);
#pragma unroll
  for (int w = 0; w < NT / 32; ++w) join(red[w * B + (tid & (B - 1))]);
}

template <int L, int B, int S>
__global__ void __launch_bounds__(fx_threads<L, B>(), fx_maxr<L>() <= 16 ? 512 / fx_threads<L, B>() : 1)
    k_fx_xy(double2 *data, long long astride, long long sj, long long so, int mz, FxTab tw) {
  constexpr int R1 = FxFac<L>::R1, R2 = FxFac<L>::R2, NT = fx_threads<L, B>();
  extern __shared__ __align__(16) unsigned char smraw[];
  fx2 *ex = reinterpret_cast<fx2 *>(smraw);  // [L][B]
  __shared__ FxSize red[NT / 32 * B];
  const int tid = threadIdx.x, b = tid & (B - 1), q = tid / B;
  const int z0 = blockIdx.x * B;
  const bool col = b < mz - z0;
  double2 *base = data + blockIdx.z * astride + (long long)blockIdx.y * so + z0 + b;
  double2 x[R2];
#pragma unroll
  for (int n2 = 0; n2 < R2; ++n2)
    x[n2] = (col && q < R1) ? base[(long long)(q + R1 * n2) * sj] : make_double2(0.0, 0.0);
  const FxScale sc = fx_scale(fx_col_size<B, NT>(fx_size(x), red, tid), 62, 64);
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
        base[(long long)(q + R2 * k1) * sj] = fx_store(u[k1], sc.out + 2, sc);
    }
  }
}

// ---------------------------------------------------------------------------
// Derivative round trips along x or y (see k_fft_xy_rt): d1 = IFFT(i k FFT(Z))
// / (L nz), d2 = IFFT(-k^2 FFT(Z)) / (L nz).  c1, c2: k / 2^e1 and -k^2 / 2^e2
// in Q62 (first derivative 0 on the Nyquist index).  ACC (the y round trip):
// the coefficient of d2 takes -kz^2 too (cz / 2^ez in Q62, brought to a common
// exponent with c2 for each column), so that d2 is the y and z part of the
// laplacian, and the x part in out1 is added.
// At 256^3: 362 us a round trip against 1359 us on the FP64 pipe, 128^3 56 us
// against 178 (344 and 53 without the products' sizes, below).  Inputs convert on
// the FP64 pipe, outputs (two per input) on the integer pipe: 375 us instead of 344
// with both on the former, 388 on the latter.
// Between the transforms each product k X, k^2 X is brought to the size that the
// inverse transform has room for: a pencil whose power lies at small k (a k^-2
// spectrum, a single wave) fills little of the coefficients' range, and with the
// spectrum's size alone (in use before) its derivatives were up to 35 times as
// far off as an FP64 round trip's at 512 points; now nowhere further.
template <int L, int B, bool ACC>
__global__ void __launch_bounds__(fx_threads<L, B>(), fx_maxr<L>() <= 16 ? 384 / fx_threads<L, B>() : 1) k_fx_rt(
    const double2 *__restrict__ in, double2 *__restrict__ out0, double2 *out1, long long sj,
    long long so, int mz, FxTab tw, const long long *__restrict__ c1,
    const long long *__restrict__ c2, const long long *__restrict__ cz, int e1, int e2, int ez) {
  constexpr int R1 = FxFac<L>::R1, R2 = FxFac<L>::R2, NT = fx_threads<L, B>();
  extern __shared__ __align__(16) unsigned char smraw[];
  fx2 *ex0 = reinterpret_cast<fx2 *>(smraw), *ex1 = ex0 + L * B;  // [L][B] each
  __shared__ FxSize size[NT / 32 * B];
  __shared__ float4 red[NT / 32 * B];
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
  const FxScale sc = fx_scale(fx_col_size<B, NT>(fx_size(x), size, tid), 62, 64);
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
  int zshift = 0;
  long long z2 = 0;
  if (ACC) {  // the column's -kz^2; c2 >> zshift and z2 at the exponent e2
    const long long v = __ldg(cz + min(z0 + b, mz - 1));
    if (v != 0) {
      const int up = max(__clzll((unsigned long long)-v) - 2, 0);
      const int e = max(e2, ez - up) + 1;
      zshift = min(e - e2, 63);
      z2 = (v << up) >> min(e - (ez - up), 63);
      e2 = e;
    }
  }
  auto coef = [&](int o, int k1) {
    const long long c = __ldg((o ? c2 : c1) + q + R2 * k1);
    return ACC && o ? (c >> zshift) + z2 : c;
  };
  // the spectrum waits in the thread's own slots of ex1 between the two
  // inverse transforms (in registers it would halve the resident CTAs).  From 16
  // points a thread on the two share their code: unrolled, the kernel waited for
  // instructions more than for anything else (128^3 57.3 -> 53.3 us, 96^3
  // 33.0 -> 31.6, 256^3 351 -> 344; 64^3 the other way, 13.5 -> 14.3).
  constexpr int kShare = R1 >= 16 || R2 >= 16 || R1 % 3 == 0 ? 1 : 2;
  auto slot = [&](int k1) { return (k1 * R2 + q) * B + b; };
  fx2 u[R1];
  float2 p = make_float2(0.0f, 0.0f);  // the sizes of the two products, units of 4
  if (q < R2) {
#pragma unroll
    for (int n1 = 0; n1 < R1; ++n1) u[n1] = ex0[fx_row<L, B>(n1 * R2 + q) * B + b];
    fx_dft<R1, -1>(u);  // u[k1] = X[q + R2 k1]
    if (z0 + b + q == 0) u[0] = fx_mk(0, 0);  // the constant: both coefficients are 0
    unsigned long long p1 = 0, p2 = 0;
#pragma unroll
    for (int k1 = 0; k1 < R1; ++k1) {
      // (|Re| + |Im| <= 2^63, a coefficient 2^62: 16 products fit)
      const unsigned long long t = ((fx_abshi(u[k1].x) + fx_abshi(u[k1].y)) >> 2) + 1;
      p1 += t * (fx_abshi(coef(0, k1)) + 1);
      p2 += t * (fx_abshi(coef(1, k1)) + 1);
      ex1[slot(k1)] = u[k1];
    }
    p = make_float2(__ull2float_ru(p1), __ull2float_ru(p2));
  }
  float2 s = p;
  fx_col_sums<B, NT>(p, s, red, tid);
  __syncthreads();  // ex0 is rewritten below (also where fx_col_sums has no barrier)
  const int room[2] = {fx_room_sum(p.x, s.x, 2, 62, 64), fx_room_sum(p.y, s.y, 2, 62, 64)};
#pragma unroll kShare
  for (int o = 0; o < 2; ++o) {
    if (q < R2) {
      const int up = max(o ? room[1] : room[0], 0), down = up - (o ? room[1] : room[0]);
#pragma unroll
      for (int k1 = 0; k1 < R1; ++k1) {
        const fx2 v = ex1[slot(k1)];
        const long long c = coef(o, k1) >> down;
        const int ch = fx_hi(c), cl = (int)c;
        const long long cx = fx_mul(v.x, ch, cl) << up, cy = fx_mul(v.y, ch, cl) << up;
        u[k1] = o ? fx_mk(cx, cy) : fx_mk(-cy, cx);  // -k^2 X, i k X
      }
      fx_dft<R1, +1>(u);
    }
    if (o) __syncthreads();  // every slot of ex1 is read
    fx2 *ex = o ? ex1 : ex0;
    if (q < R2) {
#pragma unroll
      for (int n1 = 0; n1 < R1; ++n1)
        ex[fx_row<L, B>(q * R1 + n1) * B + b] =
            n1 == 0 ? fx_quarter(u[n1]) : fx_cmul<+1>(u[n1], fx_tw(tw, n1 * q));
    }
  }
  __syncthreads();
  if (q < R1) {
    // forward twiddle, coefficient and inverse twiddle took 2 bits each
    const int e = sc.out + 6;
#pragma unroll kShare
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
          double2 r = fx_store(v[n2], e + (o ? e2 - room[1] : e1 - room[0]), sc);
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
// host side
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
    fx_split(C - S, a[4 * k + 2], a[4 * k + 3]);
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
static void fx_coefs1(std::vector<long long> &t, int L, double unit, int e1, int odd) {
  for (int k = 0; k < L; ++k) {
    const int f = k > L / 2 ? k - L : k;
    t.push_back(2 * k == L ? 0 : llrintl(ldexpl((long double)unit * f / odd, 62 - e1)));
  }
}
static void fx_coefs2(std::vector<long long> &t, int L, int count, double unit2, int e2, int odd) {
  for (int k = 0; k < count; ++k) {
    const int f = k > L / 2 ? L - k : k;
    t.push_back(-llrintl(ldexpl((long double)unit2 * f * f / odd, 62 - e2)));
  }
}
static int fx_odd(int n) {
  while (n % 2 == 0) n /= 2;
  return n;
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
  const int oz = fx_odd(g.nz), ox = fx_odd(g.nx) * oz, oy = fx_odd(g.ny) * oz;
  // of the coefficients as they are stored, with the odd parts taken out: the
  // bits that a larger exponent leaves empty are lost to the products (144x96x96
  // laplacian of white noise 8.4 -> 0.6 times the error of an FP64 round trip)
  c->fx_e[0] = fx_exp(g.kxmax / ox);
  c->fx_e[1] = fx_exp(qx / ox);
  c->fx_e[2] = fx_exp(g.kymax / oy);
  c->fx_e[3] = fx_exp(qy / oy);
  c->fx_e[4] = fx_exp(qz / oy);
  for (int e : c->fx_e)  // a box whose k leave the exponent range of the passes
    if (e < -200 || e > 200) return IH_OK;
  std::vector<long long> t;
  fx_coefs1(t, g.nx, g.kxu, c->fx_e[0], ox);
  fx_coefs2(t, g.nx, g.nx, g.kx2, c->fx_e[1], ox);
  fx_coefs1(t, g.ny, g.kyu, c->fx_e[2], oy);
  fx_coefs2(t, g.ny, g.ny, g.ky2, c->fx_e[3], oy);
  for (int k = 0; k < g.mz; ++k) {  // d/dz's kz / nz: FP64
    const double f = (double)((long double)g.kzu * k / g.nz);
    long long bits;
    memcpy(&bits, &f, sizeof f);
    t.push_back(bits);
  }
  fx_coefs2(t, g.nz, g.mz, g.kz2, c->fx_e[4], oy);
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
    const int e1 = c->fx_e[2 * axis] - scale, e2 = c->fx_e[2 * axis + 1] - scale,
              ez = c->fx_e[4] - scale;
    const size_t sm = sizeof(fx2) * L * B * 2;
    const dim3 grid((g.mz + B - 1) / B, outer);
    auto kf = axis == 1 ? k_fx_rt<L, B, true> : k_fx_rt<L, B, false>;
    want_smem(kf, sm);
    kf<<<grid, fx_threads<L, B>(), sm, c->stream>>>(z, d1, d2, sj, so, g.mz, tw, c1, c1 + L,
                                                    cz + g.mz, e1, e2, ez);
    return IH_OK;
  }
};
int fix_roundtrip(Ctx *c, const void *z, void *d1, void *d2, int axis) {
  return fx_dispatch(axis == 0 ? c->g.nx : c->g.ny,
                     FxRT{c, (const double2 *)z, (double2 *)d1, (double2 *)d2, axis});
}

}  // namespace ih
