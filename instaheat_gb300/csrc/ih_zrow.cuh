// ih_zrow.cuh -- the z engine of the fixed-point passes of the FP64 form
// (ih_fixz.cu): a row of H = nz/2 complex values (z_j = x_2j + i x_2j+1) on B
// lanes with A values each, H = A B, the structure of the wide-row engine of
// ih_zwide.cu for other lengths.
//   spectral side: lane t holds Z[t + B m], m < A;
//   real side:     lane t holds z[E t + e + A q] in register E q + e (e < E = A / B,
//                  q < B).
// One transpose through the warp's shared scratch in between; scratch columns
// are swizzled and rows padded so that the accesses of a phase (128 bytes) hit
// different banks.  Num: the arithmetic -- the complex type C, DFTs of a few
// points, the product with a table twiddle (which may take a factor 1/4, as
// quarter does) and halves.
#pragma once
#include "ih_internal.cuh"
#include "ih_fftcore.cuh"

namespace ih {

// rows of 2^a or 3 2^a points; every lane group fits a warp
template <int H> struct ZAB;
template <> struct ZAB<4> { static constexpr int A = 2, B = 2; };
template <> struct ZAB<6> { static constexpr int A = 6, B = 1; };
template <> struct ZAB<8> { static constexpr int A = 4, B = 2; };
template <> struct ZAB<12> { static constexpr int A = 6, B = 2; };
template <> struct ZAB<16> { static constexpr int A = 4, B = 4; };
template <> struct ZAB<24> { static constexpr int A = 12, B = 2; };
template <> struct ZAB<32> { static constexpr int A = 8, B = 4; };
template <> struct ZAB<48> { static constexpr int A = 12, B = 4; };
template <> struct ZAB<64> { static constexpr int A = 8, B = 8; };
template <> struct ZAB<96> { static constexpr int A = 24, B = 4; };
template <> struct ZAB<128> { static constexpr int A = 16, B = 8; };
template <> struct ZAB<192> { static constexpr int A = 24, B = 8; };
template <> struct ZAB<256> { static constexpr int A = 16, B = 16; };

template <typename Num, int H> struct ZRow {
  static constexpr int A = ZAB<H>::A, B = ZAB<H>::B, E = A / B, G = 32 / B;
  static_assert(A * B == H && E * B == A, "A B = H, B divides A");
  // scratch of a row, in values: successive rows start B values further into
  // the 128 bytes of a phase
  static constexpr int W = 128 / (int)sizeof(typename Num::C);
  static constexpr int X = A * B + ((B - A * B) % W + W) % W;
  // scratch column of (p, t)
  __device__ static __forceinline__ int col(int p, int t) { return p * B + (t ^ ((p / E) & (B - 1))); }
};

inline bool zrow_length(int h) {
  return h == 6 || h == 12 || h == 24 || h == 48 || h == 96 || h == 192 ||
         (h >= 4 && h <= 256 && (h & (h - 1)) == 0);
}

// the largest word of a row
template <int B>
__device__ __forceinline__ unsigned zrow_max(unsigned m) {
#pragma unroll
  for (int o = 1; o < B; o <<= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
  return m;
}

// spectral side -> real side, unnormalised inverse
template <typename Num, int H>
__device__ __forceinline__ void zrow_inverse(typename Num::C (&v)[ZAB<H>::A], int t,
                                             typename Num::C *xch, typename Num::Tab twh) {
  using R = ZRow<Num, H>;
  constexpr int A = R::A, B = R::B, E = R::E;
  Num::template dft<A, +1>(v);
#pragma unroll
  for (int p = 0; p < A; ++p)
    xch[R::col(p, t)] = p == 0 ? Num::quarter(v[p]) : Num::template cmul<+1>(v[p], twh, p * t);
  __syncwarp();
#pragma unroll
  for (int e = 0; e < E; ++e) {
    typename Num::C u[B];
#pragma unroll
    for (int s = 0; s < B; ++s) u[s] = xch[(E * t + e) * B + (s ^ t)];
    Num::template dft<B, +1>(u);
#pragma unroll
    for (int q = 0; q < B; ++q) v[E * q + e] = u[q];
  }
  __syncwarp();
}
// real side -> spectral side, forward
template <typename Num, int H>
__device__ __forceinline__ void zrow_forward(typename Num::C (&v)[ZAB<H>::A], int t,
                                             typename Num::C *xch, typename Num::Tab twh) {
  using R = ZRow<Num, H>;
  constexpr int A = R::A, B = R::B, E = R::E;
#pragma unroll
  for (int e = 0; e < E; ++e) {
    typename Num::C u[B];
#pragma unroll
    for (int q = 0; q < B; ++q) u[q] = v[E * q + e];
    Num::template dft<B, -1>(u);
#pragma unroll
    for (int s = 0; s < B; ++s)
      xch[(E * t + e) * B + (s ^ t)] =
          s == 0 ? Num::quarter(u[s]) : Num::template cmul<-1>(u[s], twh, (E * t + e) * s);
  }
  __syncwarp();
#pragma unroll
  for (int p = 0; p < A; ++p) v[p] = xch[R::col(p, t)];
  __syncwarp();
  Num::template dft<A, -1>(v);
}

// c2r split, in place: x[m] = X_k (k = t + B m), xH = X_H on t == 0 -> E + i O
// (times quarter's factor) with E = X_k + conj X_(H-k), O = (X_k - conj X_(H-k))
// exp(2 pi i k / nz).  X_(H-k) is register A - 1 - m of lane B - t, or register
// A - m of lane 0 itself (X_H for m = 0).  Registers m and A - 1 - m are each
// other's partners (but on lane 0), so they are formed together, before either
// is overwritten; lane 0's X_(A-m) is the register A - 1 - m of the step before.
template <typename Num, int H>
__device__ __forceinline__ void zrow_c2r_prep(typename Num::C (&x)[ZAB<H>::A], typename Num::C xH,
                                              int t, int gbase, typename Num::Tab twz) {
  using C = typename Num::C;
  constexpr int A = ZAB<H>::A, B = ZAB<H>::B;
  const int src = gbase + ((B - t) & (B - 1));
  auto split = [&](C a, C pc, int k) {
    pc.y = -pc.y;
    const C e = Num::quarter(Num::add(a, pc)),
            o = Num::template cmul<+1>(Num::sub(a, pc), twz, k);
    return Num::mk(e.x - o.y, e.y + o.x);
  };
  C prev = xH;
#pragma unroll
  for (int m = 0; m < A / 2; ++m) {
    const int n = A - 1 - m;
    C pm = Num::shfl(x[n], src), pn = Num::shfl(x[m], src);
    const C keep = x[n];
    if (t == 0) {
      pm = prev;
      pn = x[m + 1];
    }
    const C a = split(x[m], pm, t + B * m);
    x[n] = split(x[n], pn, t + B * n);
    x[m] = a;
    prev = keep;
  }
}

// r2c split: v[m] = Z_k (k = t + B m) -> X_k (times quarter's factor), xH = X_H
// on t == 0: X_k = E_k + exp(-2 pi i k / nz) O_k, E_k = (Z_k + conj Z_(H-k)) / 2,
// O_k = (Z_k - conj Z_(H-k)) / (2 i)
template <typename Num, int H>
__device__ __forceinline__ void zrow_r2c_post(typename Num::C (&v)[ZAB<H>::A], int t, int gbase,
                                              typename Num::Tab twz, typename Num::C &xH) {
  using C = typename Num::C;
  constexpr int A = ZAB<H>::A, B = ZAB<H>::B;
  const int src = gbase | ((B - t) & (B - 1));
  auto split = [&](C z, C pz, int k, C *last) {
    const C e = Num::half_quarter(Num::mk(z.x + pz.x, z.y - pz.y));
    const C o = Num::half(Num::mk(z.y + pz.y, pz.x - z.x));
    if (last) *last = Num::sub(e, Num::quarter(o));  // exp(-i pi) = -1
    return Num::add(e, Num::template cmul<-1>(o, twz, k));
  };
  C prev = v[0];  // lane 0: Z_(H - 0) = Z_0
#pragma unroll
  for (int m = 0; m < A / 2; ++m) {
    const int n = A - 1 - m;
    C pm = Num::shfl(v[n], src), pn = Num::shfl(v[m], src);
    const C keep = v[n];
    if (t == 0) {
      pm = prev;
      pn = v[m + 1];
    }
    const C a = split(v[m], pm, t + B * m, m == 0 ? &xH : nullptr);
    v[n] = split(v[n], pn, t + B * n, nullptr);
    v[m] = a;
    prev = keep;
  }
}

}  // namespace ih
