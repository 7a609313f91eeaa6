// ih_zreg.cu -- the z passes of the mixed form (FP32) for power-of-two rows of
// H = nz/2 <= 64 complex values, in registers: the operations of the warp-row
// engine (zfft_dif and the splits of ih_fft.cu), value by value, so the results
// are the same to the bit.
//
// That engine holds a row across a warp, one or two values a lane, and spends a
// stage on two shuffles and a multiplication by 1 on half of the lanes.  Here a
// row lies on B lanes with A values each, H = A B: log2 A radix-2 stages in
// registers, one exchange through shared memory, log2 B stages in registers.
//   in:  lane t holds value t + B i in register i (reals 2 j, 2 j + 1 of value j);
//   out: lane t holds frequency t + B m in register m: the bit-reversed positions
//        that end up on one lane are a lane's own again, for both directions.
#include "ih_internal.cuh"
#include "ih_fftcore.cuh"

namespace ih {

using F2 = C2<float>;

template <int H> struct RzAB;
template <> struct RzAB<4> { static constexpr int A = 2, B = 2; };
template <> struct RzAB<8> { static constexpr int A = 4, B = 2; };
template <> struct RzAB<16> { static constexpr int A = 4, B = 4; };
template <> struct RzAB<32> { static constexpr int A = 8, B = 4; };
template <> struct RzAB<64> { static constexpr int A = 8, B = 8; };

template <int H> struct RzGeo {
  static constexpr int A = RzAB<H>::A, B = RzAB<H>::B, E = A / B, G = 32 / B;
  // scratch of a row: the rows of a half-warp start B values apart mod 16
  static constexpr int X = H + B;
  // scratch place of value (i, u): the lanes of a half-warp, which write one i
  // and read one u, are on 16 different bank pairs
  __device__ static __forceinline__ int at(int i, int u) {
    const int f = E == 2 ? (B == 4 ? ((i >> 2) & 1) | (i & 2) : i >> 1) : i;
    return i * B + (u ^ (f & (B - 1)));
  }
};
__host__ __device__ constexpr int rz_brev(int k, int n) {  // of an index below n
  int r = 0;
  for (int b = 1; b < n; b <<= 1) {
    r = 2 * r + (k & 1);
    k >>= 1;
  }
  return r;
}

template <int H> struct RzTw {
  F2 t1[RzGeo<H>::A - 1];                              // stages before the exchange, lane t
  F2 t2[RzGeo<H>::B / 2 > 1 ? RzGeo<H>::B / 2 - 1 : 1];  // after: w_B^1 .. (the same on all)
  F2 wz[RzGeo<H>::A];                                  // exp(-2 pi i k / nz), k = t + B m
  __device__ __forceinline__ void load(const F2 *__restrict__ twh, const F2 *__restrict__ twz,
                                       int t) {
    constexpr int A = RzGeo<H>::A, B = RzGeo<H>::B;
    int n = 0;
#pragma unroll
    for (int half = A / 2; half >= 1; half /= 2) {
#pragma unroll
      for (int i = 0; i < half; ++i) t1[n++] = twh[(t + B * i) * (A / (2 * half))];
    }
#pragma unroll
    for (int i = 1; i < B / 2; ++i) t2[i - 1] = twh[i * A];
#pragma unroll
    for (int m = 0; m < A; ++m) wz[m] = twz[t + B * m];
  }
};
template <int S> __device__ __forceinline__ F2 rz_cj(F2 w) {
  if (S > 0) w.y = -w.y;
  return w;
}

// a b with its roundings spelled out (and those of the products of two rows below):
// the compiler contracts the plain expression one way or the other from kernel to
// kernel; these are the ways of the warp-row engine, found by comparing results.
// FIRST: a.x b.y is the product that
// is not rounded in the imaginary part, else a.y b.x.
template <bool FIRST = false> __device__ __forceinline__ F2 rz_cmul(F2 a, F2 b) {
  return mk2<float>(__fmaf_rn(a.x, b.x, -__fmul_rn(a.y, b.y)),
                    FIRST ? __fmaf_rn(a.x, b.y, __fmul_rn(a.y, b.x))
                          : __fmaf_rn(a.y, b.x, __fmul_rn(a.x, b.y)));
}

// the transform of a row, sign S
template <int S, int H>
__device__ __forceinline__ void rz_dif(F2 (&v)[RzGeo<H>::A], const RzTw<H> &w, int t, F2 *buf) {
  using Gm = RzGeo<H>;
  constexpr int A = Gm::A, B = Gm::B, E = Gm::E;
  int n = 0;
#pragma unroll
  for (int half = A / 2; half >= 1; half /= 2) {
#pragma unroll
    for (int b = 0; b < A; b += 2 * half) {
#pragma unroll
      for (int i = 0; i < half; ++i) {
        const F2 x = v[b + i], y = v[b + i + half];
        v[b + i] = cadd(x, y);
        v[b + i + half] = rz_cmul(csub(x, y), rz_cj<S>(w.t1[n + i]));
      }
    }
    n += half;
  }
#pragma unroll
  for (int i = 0; i < A; ++i) buf[Gm::at(i, t)] = v[i];
  __syncwarp();
#pragma unroll
  for (int e = 0; e < E; ++e) {
    const int i = rz_brev(t + B * e, A);
    F2 u[B];
#pragma unroll
    for (int s = 0; s < B; ++s) u[s] = buf[Gm::at(i, s)];
#pragma unroll
    for (int half = B / 2; half >= 1; half /= 2) {
#pragma unroll
      for (int b = 0; b < B; b += 2 * half) {
#pragma unroll
        for (int j = 0; j < half; ++j) {
          const F2 x = u[b + j], y = u[b + j + half];
          u[b + j] = cadd(x, y);
          const F2 d = csub(x, y);
          u[b + j + half] = j == 0 ? d : rz_cmul(d, rz_cj<S>(w.t2[j * (B / (2 * half)) - 1]));
        }
      }
    }
#pragma unroll
    for (int s = 0; s < B; ++s) v[e + E * rz_brev(s, B)] = u[s];
  }
  __syncwarp();
}

__device__ __forceinline__ F2 rz_shfl(F2 v, int src) {
  return mk2<float>(__shfl_sync(0xffffffffu, v.x, src), __shfl_sync(0xffffffffu, v.y, src));
}
// zr2c_post_lanes: Z_k -> X_k in place, xH = X_H on lane 0.  Z_(H-k) is register
// A - 1 - m of lane B - t, on lane 0 its own register A - m (Z_0 for m = 0).
template <int H>
__device__ __forceinline__ void rz_post(F2 (&v)[RzGeo<H>::A], const RzTw<H> &w, int t, int gbase,
                                        F2 &xH) {
  constexpr int A = RzGeo<H>::A, B = RzGeo<H>::B;
  const int src = gbase + ((B - t) & (B - 1));
  F2 pz[A];
#pragma unroll
  for (int m = 0; m < A; ++m) pz[m] = rz_shfl(v[A - 1 - m], src);
  if (t == 0) {
#pragma unroll
    for (int m = 0; m < A; ++m) pz[m] = v[(A - m) % A];
  }
#pragma unroll
  for (int m = 0; m < A; ++m) {
    const F2 z = v[m];
    const F2 zc = mk2<float>(pz[m].x, -pz[m].y);
    const F2 e = mk2<float>(0.5f * (z.x + zc.x), 0.5f * (z.y + zc.y));
    const F2 o = mk2<float>(0.5f * (z.y - zc.y), -0.5f * (z.x - zc.x));
    if (m == 0) xH = csub(e, o);  // exp(-i pi) = -1
    v[m] = cadd(e, rz_cmul<(H < 64)>(o, w.wz[m]));
  }
}
// zc2r_prep: X_k, X_H on lane 0 -> E + i O, in place
template <int H>
__device__ __forceinline__ void rz_prep(F2 (&x)[RzGeo<H>::A], F2 xH, const RzTw<H> &w, int t,
                                        int gbase) {
  constexpr int A = RzGeo<H>::A, B = RzGeo<H>::B;
  const int src = gbase + ((B - t) & (B - 1));
  F2 pc[A];
#pragma unroll
  for (int m = 0; m < A; ++m) pc[m] = rz_shfl(x[A - 1 - m], src);
  if (t == 0) {
#pragma unroll
    for (int m = 0; m < A; ++m) pc[m] = m == 0 ? xH : x[A - m];
  }
#pragma unroll
  for (int m = 0; m < A; ++m) {
    pc[m].y = -pc[m].y;  // conj X_(H-k)
    const F2 e = cadd(x[m], pc[m]), d = csub(x[m], pc[m]);
    const F2 o = rz_cmul(d, rz_cj<+1>(w.wz[m]));
    x[m] = mk2<float>(e.x - o.y, e.y + o.x);
  }
}
template <int H>
__device__ __forceinline__ void rz_fetch(const F2 *row, int t, bool valid, F2 (&x)[RzGeo<H>::A],
                                         F2 &xH) {
#pragma unroll
  for (int m = 0; m < RzGeo<H>::A; ++m)
    x[m] = valid ? row[t + RzGeo<H>::B * m] : mk2<float>(0, 0);
  xH = (valid && t == 0) ? row[H] : mk2<float>(0, 0);
}
template <int H>
__device__ __forceinline__ void rz_store(const F2 (&v)[RzGeo<H>::A], F2 xH, int t, bool valid,
                                         F2 *row) {
  if (!valid) return;
#pragma unroll
  for (int m = 0; m < RzGeo<H>::A; ++m) row[t + RzGeo<H>::B * m] = v[m];
  if (t == 0) row[H] = xH;
}

constexpr int kRzWarps = 4;
struct RzLane {
  int t, gbase;
  bool valid;
  long long row;
  F2 *buf;
};
template <int H>
__device__ __forceinline__ RzLane rz_lane(long long group, long long rows, F2 *buf) {
  using Gm = RzGeo<H>;
  const int lane = threadIdx.x & 31, grp = lane / Gm::B;
  RzLane ln;
  ln.t = lane & (Gm::B - 1);
  ln.gbase = lane & ~(Gm::B - 1);
  ln.row = group * Gm::G + grp;
  ln.valid = ln.row < rows;
  ln.buf = buf + grp * Gm::X;
  return ln;
}

template <int H, bool FORWARD>
__global__ void __launch_bounds__(32 * kRzWarps) k_rz_pass(
    const float *__restrict__ in, long long istride, float *__restrict__ out, long long ostride,
    long long rows, const F2 *__restrict__ twh, const F2 *__restrict__ twz) {
  using Gm = RzGeo<H>;
  __shared__ F2 xs[kRzWarps][Gm::G * Gm::X];
  const int warp = threadIdx.x >> 5;
  const RzLane ln = rz_lane<H>((long long)blockIdx.x * kRzWarps + warp, rows, xs[warp]);
  RzTw<H> w;
  w.load(twh, twz, ln.t);
  F2 v[Gm::A], xH;
  if (FORWARD) {
    const F2 *src = reinterpret_cast<const F2 *>(in + blockIdx.y * istride) + ln.row * H;
#pragma unroll
    for (int i = 0; i < Gm::A; ++i) v[i] = ln.valid ? src[ln.t + Gm::B * i] : mk2<float>(0, 0);
    rz_dif<-1, H>(v, w, ln.t, ln.buf);
    rz_post<H>(v, w, ln.t, ln.gbase, xH);
    rz_store<H>(v, xH, ln.t, ln.valid,
                reinterpret_cast<F2 *>(out) + blockIdx.y * ostride + ln.row * (H + 1));
  } else {
    rz_fetch<H>(reinterpret_cast<const F2 *>(in) + blockIdx.y * istride + ln.row * (H + 1), ln.t,
                ln.valid, v, xH);
    rz_prep<H>(v, xH, w, ln.t, ln.gbase);
    rz_dif<+1, H>(v, w, ln.t, ln.buf);
    F2 *dst = reinterpret_cast<F2 *>(out + blockIdx.y * ostride) + ln.row * H;
    if (ln.valid) {
#pragma unroll
      for (int i = 0; i < Gm::A; ++i) dst[ln.t + Gm::B * i] = v[i];
    }
  }
}

// ---------------------------------------------------------------------------
// The fused last z pass of the RHS (k_fft_z_rhs_fused, ih_fft.cu), from its
// parts: a derivative row, rho and p of a point, the transform of a product
struct RzIn {
  const F2 *d4;
  long long dstride;
  float kzu, invnz;
  int zsrc;  // d/dz from Z in slot 4
};
template <int H>
__device__ __forceinline__ void rz_deriv(const RzIn &in, int a, const RzLane &ln, const RzTw<H> &w,
                                         F2 (&v)[RzGeo<H>::A]) {
  constexpr int A = RzGeo<H>::A, B = RzGeo<H>::B;
  F2 xH;
  const bool z = in.zsrc && a == 2;
  rz_fetch<H>(in.d4 + (z ? 4 : a) * in.dstride + ln.row * (H + 1), ln.t, ln.valid, v, xH);
  if (z) {  // i kz Z / nz, zero on the Nyquist index
#pragma unroll
    for (int m = 0; m < A; ++m) {
      const float f = kfac<float>(in.kzu, ln.t + B * m) * in.invnz;
      v[m] = mk2<float>(-v[m].y * f, v[m].x * f);
    }
    xH = mk2<float>(0, 0);
  }
  rz_prep<H>(v, xH, w, ln.t, ln.gbase);
  rz_dif<+1, H>(v, w, ln.t, ln.buf);
}
struct RzPoint {
  const float *yfl;
  float *p, *rho;
  long long N;
  float inv_a2, m2, third, phib, pib, psib;
  __device__ __forceinline__ void init(const double *ysc, float mass2) {
    const double a = ysc[4];
    inv_a2 = (float)(1.0 / (a * a));
    m2 = mass2;
    third = (float)(1.0 / 3.0);
    phib = (float)ysc[0];
    pib = (float)ysc[1];
    psib = (float)ysc[2];
  }
  // value j of a row; its rho and p added to sr, sp
  template <int H>
  __device__ __forceinline__ void at(const RzLane &ln, int j, F2 dx, F2 dy, F2 dz, float &sr,
                                     float &sp) const {
    const long long e = ln.row * (2 * H) + 2 * j;
    const F2 phi = *reinterpret_cast<const F2 *>(yfl + e);
    const F2 dph = *reinterpret_cast<const F2 *>(yfl + N + e);
    const F2 ps = *reinterpret_cast<const F2 *>(yfl + 2 * N + e);
    F2 r, q;
    rho_p<float, true>(dx.x, dy.x, dz.x, phi.x, dph.x, ps.x, inv_a2, m2, third, phib, pib, psib,
                       r.x, q.x);
    rho_p<float, true>(dx.y, dy.y, dz.y, phi.y, dph.y, ps.y, inv_a2, m2, third, phib, pib, psib,
                       r.y, q.y);
    *reinterpret_cast<F2 *>(p + e) = q;
    if (rho) *reinterpret_cast<F2 *>(rho + e) = r;
    sr += r.x + r.y;
    sp += q.x + q.y;
  }
};
// the values whose rho and p are added in FP32 before the FP64 sums: j and j + 32
// of a row of 64 (one lane's of the warp-row engine), else single ones
template <int H> constexpr int kRzPair = H == 64 ? 2 : 1;
// the product of two rows -> its half spectrum
template <int H>
__device__ __forceinline__ void rz_product(const F2 (&x)[RzGeo<H>::A], const F2 (&y)[RzGeo<H>::A],
                                           const RzTw<H> &w, const RzLane &ln, F2 *spec) {
  constexpr int A = RzGeo<H>::A;
  F2 u[A], xH;
#pragma unroll
  for (int i = 0; i < A; ++i)
    u[i] = mk2<float>(__fmul_rn(x[i].x, y[i].x), __fmul_rn(x[i].y, y[i].y));
  rz_dif<-1, H>(u, w, ln.t, ln.buf);
  rz_post<H>(u, w, ln.t, ln.gbase, xH);
  rz_store<H>(u, xH, ln.t, ln.valid, spec + ln.row * (H + 1));
}
template <int H>
__device__ __forceinline__ void rz_lap(const F2 (&v)[RzGeo<H>::A], const RzLane &ln, float *lap) {
  if (!ln.valid) return;
#pragma unroll
  for (int i = 0; i < RzGeo<H>::A; ++i)
    *reinterpret_cast<F2 *>(lap + ln.row * (2 * H) + 2 * (ln.t + RzGeo<H>::B * i)) = v[i];
}

// A warp per group of rows.  The warp-row engine was bound by its instructions
// (2.8 a clock and SM); 128^3 59.7 -> 40.2 us, 64^3 18.3 -> 15.9.  CTAs per SM 3 / 4 /
// 5 at 128^3: 50.0 / 40.2 / 46.0 us (the last spills).
template <int H>
__global__ void __launch_bounds__(32 * kRzWarps, 4) k_rz_rhs(
    const RzIn in, RzPoint pt, const double *ysc, float mass2, float *lap, F2 *s6,
    long long sstride, int gw, double *partials, long long rows, const F2 *__restrict__ twh,
    const F2 *__restrict__ twz) {
  using Gm = RzGeo<H>;
  constexpr int A = Gm::A, B = Gm::B;
  __shared__ F2 xs[kRzWarps][Gm::G * Gm::X];
  const int warp = threadIdx.x >> 5;
  const RzLane ln = rz_lane<H>((long long)blockIdx.x * kRzWarps + warp, rows, xs[warp]);
  RzTw<H> w;
  w.load(twh, twz, ln.t);
  F2 d[3][A];
  {
    F2 v[A];
    rz_deriv<H>(in, 3, ln, w, v);
    rz_lap<H>(v, ln, lap);
  }
#pragma unroll
  for (int a = 0; a < 3; ++a) rz_deriv<H>(in, a, ln, w, d[a]);
  pt.init(ysc, mass2);
  double dr = 0.0, dp = 0.0;
  if (ln.valid) {
    constexpr int P = kRzPair<H>;
#pragma unroll
    for (int m = 0; m < A / P; ++m) {
      float sr = 0, sp = 0;
#pragma unroll
      for (int q = 0; q < P; ++q) {
        const int i = m + q * (A / P);
        pt.at<H>(ln, ln.t + B * i, d[0][i], d[1][i], d[2][i], sr, sp);
      }
      dr += (double)sr;
      dp += (double)sp;
    }
  }
  rhs_partial<32 * kRzWarps>(dr, dp, partials);
  if (!gw) return;
  int pr = 0;
#pragma unroll
  for (int a = 0; a < 3; ++a) {
#pragma unroll
    for (int b = a; b < 3; ++b, ++pr) {
      rz_product<H>(d[a], d[b], w, ln, s6 + pr * sstride);
    }
  }
}

// eight warps per group of rows, for grids with few rows: four transform the
// derivatives, then six the products and two take half the points each.  One warp
// a group / eight, by groups: 16 (16^3) 10.2 / 7.9 us, 128 (32^3) 10.2 / 8.1, 512
// (64^3) 15.9 / 17.1, 1024 (128x64x64) 18.1 / 22.5.
template <int H> struct RzCo {
  F2 xs[6][RzGeo<H>::G * RzGeo<H>::X];
  F2 d[3][RzGeo<H>::A][32];
};
template <int H>
__global__ void __launch_bounds__(256) k_rz_rhs_co(
    const RzIn in, RzPoint pt, const double *ysc, float mass2, float *lap, F2 *s6,
    long long sstride, int gw, double *partials, long long rows, const F2 *__restrict__ twh,
    const F2 *__restrict__ twz) {
  using Gm = RzGeo<H>;
  constexpr int A = Gm::A, B = Gm::B, P = kRzPair<H>;
  __shared__ RzCo<H> sm;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const RzLane ln = rz_lane<H>(blockIdx.x, rows, sm.xs[warp < 6 ? warp : 0]);
  RzTw<H> w;
  if (warp < 6) w.load(twh, twz, ln.t);
  if (warp < 4) {
    F2 v[A];
    rz_deriv<H>(in, warp, ln, w, v);
    if (warp == 3) {
      rz_lap<H>(v, ln, lap);
    } else {
#pragma unroll
      for (int i = 0; i < A; ++i) sm.d[warp][i][lane] = v[i];
    }
  }
  __syncthreads();
  double dr = 0.0, dp = 0.0;
  if (warp >= 6) {
    pt.init(ysc, mass2);
    if (ln.valid) {
#pragma unroll
      for (int m0 = 0; m0 < A / P / 2; ++m0) {
        const int m = m0 + (warp - 6) * (A / P / 2);
        float sr = 0, sp = 0;
#pragma unroll
        for (int q = 0; q < P; ++q) {
          const int i = m + q * (A / P);
          pt.at<H>(ln, ln.t + B * i, sm.d[0][i][lane], sm.d[1][i][lane], sm.d[2][i][lane], sr, sp);
        }
        dr += (double)sr;
        dp += (double)sp;
      }
    }
  } else if (gw) {
    const int ia = warp < 3 ? 0 : (warp < 5 ? 1 : 2), ib = warp < 3 ? warp : (warp < 5 ? warp - 2 : 2);
    F2 x[A], y[A];
#pragma unroll
    for (int i = 0; i < A; ++i) {
      x[i] = sm.d[ia][i][lane];
      y[i] = sm.d[ib][i][lane];
    }
    rz_product<H>(x, y, w, ln, s6 + warp * sstride);
  }
  rhs_partial<256>(dr, dp, partials);
}

// ---------------------------------------------------------------------------
// host side
bool zreg_ok(const Ctx *c) {
  return c->mixed && (c->g.h & (c->g.h - 1)) == 0 && c->g.h >= 4 && c->g.h <= 64;
}

template <typename F>
static int rz_dispatch(int H, F &&f) {
  switch (H) {
    case 4: return f.template run<4>();
    case 8: return f.template run<8>();
    case 16: return f.template run<16>();
    case 32: return f.template run<32>();
    case 64: return f.template run<64>();
    default: return IH_ERR_ARG;
  }
}
struct RzPass {
  Ctx *c;
  const void *in;
  long long istride;
  void *out;
  long long ostride;
  int count;
  bool forward;
  template <int H>
  int run() {
    const long long rows = (long long)c->g.nx * c->g.ny, per = kRzWarps * RzGeo<H>::G;
    const dim3 grid((unsigned)((rows + per - 1) / per), count);
    auto kf = forward ? k_rz_pass<H, true> : k_rz_pass<H, false>;
    kf<<<grid, 32 * kRzWarps, 0, c->stream>>>((const float *)in, istride, (float *)out, ostride,
                                              rows, (const F2 *)c->tw_h, (const F2 *)c->tw_z);
    return IH_OK;
  }
};
int zreg_pass(Ctx *c, const void *in, long long istride, void *out, long long ostride, int count,
              bool forward) {
  return rz_dispatch(c->g.h, RzPass{c, in, istride, out, ostride, count, forward});
}
struct RzRhs {
  Ctx *c;
  const void *d4, *yfl;
  const double *ysc;
  void *lap, *p, *rho, *s6;
  int gw;
  double *partials;
  int zsrc;
  template <int H>
  int run() {
    const Geom &g = c->g;
    const long long rows = (long long)g.nx * g.ny, groups = (rows + RzGeo<H>::G - 1) / RzGeo<H>::G;
    const bool co = groups <= 2LL * c->num_sms;  // see k_rz_rhs_co
    const unsigned nblk = (unsigned)(co ? groups : (groups + kRzWarps - 1) / kRzWarps);
    if (2LL * nblk > c->partials_cap) {
      c->err = "grid too large for the RHS partial-sum buffer";
      return IH_ERR_ARG;
    }
    const RzIn in{(const F2 *)d4, g.M, (float)g.kzu, (float)(1.0 / (double)g.nz), zsrc};
    RzPoint pt{};
    pt.yfl = (const float *)yfl;
    pt.p = (float *)p;
    pt.rho = (float *)rho;
    pt.N = g.N;
    const float mass2 = (float)(g.mass * g.mass);
    const F2 *th = (const F2 *)c->tw_h, *tz = (const F2 *)c->tw_z;
    c->z_blocks = (int)nblk;
    if (co)
      k_rz_rhs_co<H><<<nblk, 256, 0, c->stream>>>(in, pt, ysc, mass2, (float *)lap, (F2 *)s6, g.M,
                                                  gw, partials, rows, th, tz);
    else
      k_rz_rhs<H><<<nblk, 32 * kRzWarps, 0, c->stream>>>(in, pt, ysc, mass2, (float *)lap, (F2 *)s6,
                                                         g.M, gw, partials, rows, th, tz);
    return IH_OK;
  }
};
int zreg_rhs(Ctx *c, const void *d4, const void *yfl, const double *ysc, void *lap, void *p,
             void *rho, void *s6, int gw, double *partials, int zsrc) {
  return rz_dispatch(c->g.h, RzRhs{c, d4, yfl, ysc, lap, p, rho, s6, gw, partials, zsrc});
}

}  // namespace ih
