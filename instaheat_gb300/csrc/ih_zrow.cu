// ih_zrow.cu -- the FP32 z passes of the mixed form on the row engine of
// ih_zrow.cuh, for power-of-two rows (nz = 256 has its own kernel,
// ih_zwide.cu).  Same inputs, outputs and partial sums as the warp-per-row
// kernels of ih_fft.cu.
#include "ih_internal.cuh"
#include "ih_fftcore.cuh"
#include "ih_zrow.cuh"

namespace ih {

struct NumF {
  using C = float2;
  using Tab = const float2 *;
  __device__ static __forceinline__ C mk(float x, float y) { return make_float2(x, y); }
  __device__ static __forceinline__ C add(C a, C b) { return cadd(a, b); }
  __device__ static __forceinline__ C sub(C a, C b) { return csub(a, b); }
  __device__ static __forceinline__ C quarter(C v) { return v; }
  __device__ static __forceinline__ C half(C v) { return make_float2(0.5f * v.x, 0.5f * v.y); }
  __device__ static __forceinline__ C half_quarter(C v) { return half(v); }
  template <int S>
  __device__ static __forceinline__ C cmul(C v, Tab t, int i) {
    return ih::cmul(v, cj<S>(__ldg(t + i)));
  }
  template <int R, int S>
  __device__ static __forceinline__ void dft(C (&v)[R]) { reg_dft<float, R>(v, nullptr, 0, S); }
  __device__ static __forceinline__ C shfl(C v, int src) { return shfl_idx_c(v, src); }
};
constexpr int kZrWarps = 4;

template <int H>
__global__ void __launch_bounds__(32 * kZrWarps) k_zrow_r2c(
    const float *__restrict__ in, long long istride, float2 *__restrict__ out, long long ostride,
    long long rows, const float2 *__restrict__ twh, const float2 *__restrict__ twz) {
  using G = ZRow<NumF, H>;
  constexpr int A = G::A, B = G::B, E = G::E;
  __shared__ float2 xs[kZrWarps][G::G * G::X];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int t = lane & (B - 1), grp = lane / B, gbase = lane & ~(B - 1);
  const long long row = ((long long)blockIdx.x * kZrWarps + warp) * G::G + grp;
  const bool valid = row < rows;
  const float2 *src = reinterpret_cast<const float2 *>(in + blockIdx.y * istride) + row * H;
  float2 v[A], xH;
#pragma unroll
  for (int q = 0; q < B; ++q) {
#pragma unroll
    for (int e = 0; e < E; ++e)
      v[E * q + e] = valid ? src[E * t + e + A * q] : make_float2(0.f, 0.f);
  }
  zrow_forward<NumF, H>(v, t, &xs[warp][grp * G::X], twh);
  zrow_r2c_post<NumF, H>(v, t, gbase, twz, xH);
  if (valid) {
    float2 *dst = out + blockIdx.y * ostride + row * (H + 1);
#pragma unroll
    for (int m = 0; m < A; ++m) dst[t + B * m] = v[m];
    if (t == 0) dst[H] = xH;
  }
}

// fetch a half-spectrum row: x[m] = X_(t + B m), xH = X_H on lane 0
template <int H>
__device__ __forceinline__ void zr_fetch(const float2 *row, int t, bool valid,
                                         float2 (&x)[ZAB<H>::A], float2 &xH) {
#pragma unroll
  for (int m = 0; m < ZAB<H>::A; ++m)
    x[m] = valid ? row[t + ZAB<H>::B * m] : make_float2(0.f, 0.f);
  xH = (valid && t == 0) ? row[H] : make_float2(0.f, 0.f);
}

template <int H>
__global__ void __launch_bounds__(32 * kZrWarps) k_zrow_c2r(
    const float2 *__restrict__ in, long long istride, float *__restrict__ out, long long ostride,
    long long rows, const float2 *__restrict__ twh, const float2 *__restrict__ twz) {
  using G = ZRow<NumF, H>;
  constexpr int A = G::A, B = G::B, E = G::E;
  __shared__ float2 xs[kZrWarps][G::G * G::X];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int t = lane & (B - 1), grp = lane / B, gbase = lane & ~(B - 1);
  const long long row = ((long long)blockIdx.x * kZrWarps + warp) * G::G + grp;
  const bool valid = row < rows;
  float2 v[A], xH;
  zr_fetch<H>(in + blockIdx.y * istride + row * (H + 1), t, valid, v, xH);
  zrow_c2r_prep<NumF, H>(v, xH, t, gbase, twz);
  zrow_inverse<NumF, H>(v, t, &xs[warp][grp * G::X], twh);
  if (valid) {
    float2 *dst = reinterpret_cast<float2 *>(out + blockIdx.y * ostride) + row * H;
#pragma unroll
    for (int q = 0; q < B; ++q) {
#pragma unroll
      for (int e = 0; e < E; ++e) dst[E * t + e + A * q] = v[E * q + e];
    }
  }
}

// The fused last z pass of the RHS (see k_fft_z_rhs_fused, ih_fft.cu): d/dx and
// d/dy wait in a thread-private shared slab, d/dz in registers; one copy of the
// transform code for the four inverse and one for the six forward transforms.
template <int H> struct ZrSmem {
  float2 xs[kZrWarps][ZRow<NumF, H>::G * ZRow<NumF, H>::X];
  float2 grad[kZrWarps][2][ZAB<H>::A][32];
};

template <int H, bool ZSRC>
__global__ void __launch_bounds__(32 * kZrWarps, ZAB<H>::A <= 12 ? 6 : 4) k_zrow_rhs(
    const float2 *d4, long long dstride, const float *__restrict__ yfl, const double *ysc,
    float *lap, float *pout, float *rhoout, float2 *s6, long long sstride, int gw,
    double *partials, Geom g, const float2 *__restrict__ twh,
    const float2 *__restrict__ twz) {
  using G = ZRow<NumF, H>;
  constexpr int A = G::A, B = G::B, E = G::E;
  extern __shared__ __align__(16) unsigned char smraw[];
  ZrSmem<H> &sm = *reinterpret_cast<ZrSmem<H> *>(smraw);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int t = lane & (B - 1), grp = lane / B, gbase = lane & ~(B - 1);
  const long long rows = (long long)g.nx * g.ny;
  const long long row = ((long long)blockIdx.x * kZrWarps + warp) * G::G + grp;
  const bool valid = row < rows;
  float2 *xch = &sm.xs[warp][grp * G::X];
  const float invnz = (float)(1.0 / (double)g.nz);
  float2 dz[A];
#pragma unroll 1
  for (int i = 0; i < 4; ++i) {
    const int a = (i + 3) & 3;  // the laplacian, then d/dx, d/dy, d/dz
    float2 v[A], vH;
    zr_fetch<H>(d4 + (ZSRC && a == 2 ? 4 : a) * dstride + row * (H + 1), t, valid, v, vH);
    if (ZSRC && a == 2) {  // i kz Z / nz, zero on the Nyquist index
#pragma unroll
      for (int m = 0; m < A; ++m) {
        const float f = kfac<float>(g.kzu, t + B * m) * invnz;
        v[m] = make_float2(-v[m].y * f, v[m].x * f);
      }
      vH = make_float2(0.f, 0.f);
    }
    zrow_c2r_prep<NumF, H>(v, vH, t, gbase, twz);
    zrow_inverse<NumF, H>(v, t, xch, twh);
    if (a == 3) {
      if (valid) {
        float2 *dst = reinterpret_cast<float2 *>(lap) + row * H;
#pragma unroll
        for (int q = 0; q < B; ++q) {
#pragma unroll
          for (int e = 0; e < E; ++e) dst[E * t + e + A * q] = v[E * q + e];
        }
      }
    } else if (a < 2) {
#pragma unroll
      for (int m = 0; m < A; ++m) sm.grad[warp][a][m][lane] = v[m];
    } else {
#pragma unroll
      for (int m = 0; m < A; ++m) dz[m] = v[m];
    }
  }

  // energy density and pressure, FP64 sums of pairs of points
  const double a_sc = ysc[4];
  const float inv_a2 = (float)(1.0 / (a_sc * a_sc));
  const float m2 = (float)(g.mass * g.mass), third = (float)(1.0 / 3.0);
  const float phib = (float)ysc[0], pib = (float)ysc[1], psib = (float)ysc[2];
  const long long N2 = g.N / 2;
  double dr = 0.0, dp = 0.0;
  if (valid) {
    const float2 *yp = reinterpret_cast<const float2 *>(yfl) + row * H;
    float2 *po = reinterpret_cast<float2 *>(pout) + row * H;
#pragma unroll
    for (int q = 0; q < B; ++q) {
      float sr = 0.f, sp = 0.f;  // E pairs in FP32, as neighbours in memory
#pragma unroll
      for (int e = 0; e < E; ++e) {
        const int i = E * q + e;
        const long long at = E * t + e + A * q;
        const float2 ph = yp[at], dph = yp[N2 + at], ps = yp[2 * N2 + at];
        const float2 gx = sm.grad[warp][0][i][lane], gy = sm.grad[warp][1][i][lane];
        float2 rho, p;
        rho_p<float, true>(gx.x, gy.x, dz[i].x, ph.x, dph.x, ps.x, inv_a2, m2, third, phib, pib,
                           psib, rho.x, p.x);
        rho_p<float, true>(gx.y, gy.y, dz[i].y, ph.y, dph.y, ps.y, inv_a2, m2, third, phib, pib,
                           psib, rho.y, p.y);
        po[at] = p;
        if (rhoout) reinterpret_cast<float2 *>(rhoout)[row * H + at] = rho;
        sr += rho.x + rho.y;
        sp += p.x + p.y;
        if (e % 2 == 1 || e == E - 1) {  // at most four points in FP32
          dr += (double)sr;
          dp += (double)sp;
          sr = sp = 0.f;
        }
      }
    }
  }
  rhs_partial<32 * kZrWarps>(dr, dp, partials);
  if (!gw) return;

  // the six products d_i phi d_j phi and their forward transforms
#pragma unroll 1
  for (int pr = 0; pr < 6; ++pr) {
    const int ia = pr < 3 ? 0 : (pr < 5 ? 1 : 2);
    const int ib = pr < 3 ? pr : (pr < 5 ? pr - 2 : 2);
    float2 v[A], xH;
#pragma unroll
    for (int m = 0; m < A; ++m) {
      const float2 a = ia < 2 ? sm.grad[warp][ia][m][lane] : dz[m];
      const float2 b = ib < 2 ? sm.grad[warp][ib][m][lane] : dz[m];
      v[m] = make_float2(a.x * b.x, a.y * b.y);
    }
    zrow_forward<NumF, H>(v, t, xch, twh);
    zrow_r2c_post<NumF, H>(v, t, gbase, twz, xH);
    if (valid) {
      float2 *dst = s6 + pr * sstride + row * (H + 1);
#pragma unroll
      for (int m = 0; m < A; ++m) dst[t + B * m] = v[m];
      if (t == 0) dst[H] = xH;
    }
  }
}

// ---------------------------------------------------------------------------
template <typename F>
static int zr_dispatch(int H, F &&f) {
  switch (H) {
    case 4: return f.template run<4>();
    case 8: return f.template run<8>();
    case 16: return f.template run<16>();
    case 32: return f.template run<32>();
    case 64: return f.template run<64>();
    case 256: return f.template run<256>();
    default: return IH_ERR_ARG;
  }
}

bool zrow_ok(const Ctx *c) {
  const int h = c->g.h;
  return c->mixed && c->zwide && h >= 4 && h <= 256 && h != 128 && (h & (h - 1)) == 0;
}

struct ZrPass {
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
    const long long rows = (long long)g.nx * g.ny, per = kZrWarps * ZRow<NumF, H>::G;
    const dim3 grid((unsigned)((rows + per - 1) / per), count);
    const float2 *th = (const float2 *)c->tw_h, *tz = (const float2 *)c->tw_z;
    if (forward)
      k_zrow_r2c<H><<<grid, 32 * kZrWarps, 0, c->stream>>>((const float *)in, istride,
                                                           (float2 *)out, ostride, rows, th, tz);
    else
      k_zrow_c2r<H><<<grid, 32 * kZrWarps, 0, c->stream>>>((const float2 *)in, istride,
                                                           (float *)out, ostride, rows, th, tz);
    return IH_OK;
  }
};
int zrow_pass(Ctx *c, const void *in, long long istride, void *out, long long ostride, int count,
              bool forward) {
  return zr_dispatch(c->g.h, ZrPass{c, in, istride, out, ostride, count, forward});
}

struct ZrRhs {
  Ctx *c;
  const float2 *d4;
  const float *yfl;
  const double *ysc;
  float *lap, *p, *rho;
  float2 *s6;
  int gw;
  double *partials;
  int zsrc;
  template <int H>
  int run() {
    const Geom &g = c->g;
    const long long rows = (long long)g.nx * g.ny, per = kZrWarps * ZRow<NumF, H>::G;
    const unsigned nblk = (unsigned)((rows + per - 1) / per);
    if (2LL * nblk > c->partials_cap) {
      c->err = "grid too large for the RHS partial-sum buffer";
      return IH_ERR_ARG;
    }
    auto kf = zsrc ? k_zrow_rhs<H, true> : k_zrow_rhs<H, false>;
    const size_t sm = sizeof(ZrSmem<H>);
    want_smem(kf, sm);
    c->z_blocks = (int)nblk;
    kf<<<nblk, 32 * kZrWarps, sm, c->stream>>>(d4, g.M, yfl, ysc, lap, p, rho, s6, g.M, gw,
                                               partials, g, (const float2 *)c->tw_h,
                                               (const float2 *)c->tw_z);
    return IH_OK;
  }
};
int zrow_rhs(Ctx *c, const void *d4, const void *yfl, const double *ysc, void *lap, void *p,
             void *rho, void *s6, int gw, double *partials, int zsrc) {
  return zr_dispatch(c->g.h, ZrRhs{c, (const float2 *)d4, (const float *)yfl, ysc, (float *)lap,
                                   (float *)p, (float *)rho, (float2 *)s6, gw, partials, zsrc});
}

}  // namespace ih
