// In-register DFTs of two sequences at once in planar pairs: a PairC holds the
// real parts of two adjacent columns in one FP32x2 register pair and their
// imaginary parts in another, so every butterfly and twiddle of both columns
// is one packed instruction (fma.rn.f32x2 and its add and mul forms; sm_100
// and later).  Each lane rounds as the scalar forms of fft.cuh do.
//
// Packed FP32 has the scalar forms' FLOP rate on GB300 (measured: 36.9 T
// element operations/s for FFMA, 34.2 T for the packed form, 37.7 T for the
// packed add and mul at 16 warps per SM), so what the pairs save is issue
// slots: a 16-point DFT of two columns takes about 160 instructions where two
// scalar-complex DFTs with packed adds alone took 230.
#pragma once

#include "fft.cuh"

namespace gbn {

struct PairC {
  float2 re, im;  // columns 2j and 2j + 1
};

__device__ __forceinline__ float2 p2(float v) { return make_float2(v, v); }
__device__ __forceinline__ float2 p2neg(float2 a) { return make_float2(-a.x, -a.y); }
__device__ __forceinline__ PairC pc_add(const PairC& a, const PairC& b) {
  return PairC{__fadd2_rn(a.re, b.re), __fadd2_rn(a.im, b.im)};
}
__device__ __forceinline__ PairC pc_sub(const PairC& a, const PairC& b) {
  return PairC{__fadd2_rn(a.re, p2neg(b.re)), __fadd2_rn(a.im, p2neg(b.im))};
}
// a * (c + i s) with c and s splat over the pair
__device__ __forceinline__ PairC pc_mul(const PairC& a, float2 c, float2 s) {
  return PairC{__ffma2_rn(a.re, c, __fmul2_rn(a.im, p2neg(s))), __ffma2_rn(a.re, s, __fmul2_rn(a.im, c))};
}

// multiply by the compile-time forward twiddle w_N^J (as twc of fft.cuh)
template <int N, int J>
__device__ __forceinline__ PairC pc_twc(const PairC& a) {
  constexpr int j = ((J % N) + N) % N;
  if constexpr (j == 0) {
    return a;
  } else if constexpr (2 * j == N) {
    return PairC{p2neg(a.re), p2neg(a.im)};
  } else if constexpr (4 * j == N) {
    return PairC{a.im, p2neg(a.re)};
  } else if constexpr (4 * j == 3 * N) {
    return PairC{p2neg(a.im), a.re};
  } else {
    constexpr float c = float(cx_cos2pi(j, N));
    constexpr float s = -float(cx_sin2pi(j, N));
    return PairC{__ffma2_rn(a.re, p2(c), __fmul2_rn(a.im, p2(-s))), __ffma2_rn(a.re, p2(s), __fmul2_rn(a.im, p2(c)))};
  }
}

// forward DFT of N points of both columns, natural order in and out (dft of fft.cuh)
template <int N>
__device__ __forceinline__ void pair_dft(PairC* a) {
  if constexpr (N == 1) {
  } else if constexpr (N == 2) {
    const PairC t = a[1];
    a[1] = pc_sub(a[0], t);
    a[0] = pc_add(a[0], t);
  } else if constexpr (N == 4) {
    const PairC s02 = pc_add(a[0], a[2]), d02 = pc_sub(a[0], a[2]);
    const PairC s13 = pc_add(a[1], a[3]), d13 = pc_sub(a[1], a[3]);
    a[0] = pc_add(s02, s13);
    a[2] = pc_sub(s02, s13);
    // d02 -/+ i d13: (re + d13.im, im - d13.re) and the mirror
    a[1] = PairC{__fadd2_rn(d02.re, d13.im), __fadd2_rn(d02.im, p2neg(d13.re))};
    a[3] = PairC{__fadd2_rn(d02.re, p2neg(d13.im)), __fadd2_rn(d02.im, d13.re)};
  } else if constexpr (N == 3 || N == 5 || N == 7) {
    constexpr int M = (N - 1) / 2;
    PairC sp[M], sm[M], x0 = a[0];
    sfor<0, M>([&](auto mc) {
      constexpr int m = decltype(mc)::value;
      sp[m] = pc_add(a[m + 1], a[N - 1 - m]);
      sm[m] = pc_sub(a[m + 1], a[N - 1 - m]);
      x0 = pc_add(x0, sp[m]);
    });
    PairC out[N];
    out[0] = x0;
    sfor<1, M + 1>([&](auto kc) {
      constexpr int k = decltype(kc)::value;
      PairC re = a[0], im{};
      sfor<0, M>([&](auto mc) {
        constexpr int m = decltype(mc)::value;
        constexpr float c = float(cx_cos2pi((m + 1) * k, N));
        constexpr float s = float(cx_sin2pi((m + 1) * k, N));
        re.re = __ffma2_rn(p2(c), sp[m].re, re.re);
        re.im = __ffma2_rn(p2(c), sp[m].im, re.im);
        if constexpr (m == 0) {
          im.re = __fmul2_rn(p2(s), sm[m].re);
          im.im = __fmul2_rn(p2(s), sm[m].im);
        } else {
          im.re = __ffma2_rn(p2(s), sm[m].re, im.re);
          im.im = __ffma2_rn(p2(s), sm[m].im, im.im);
        }
      });
      // X_k = re - i im, X_{N-k} = re + i im
      out[k] = PairC{__fadd2_rn(re.re, im.im), __fadd2_rn(re.im, p2neg(im.re))};
      out[N - k] = PairC{__fadd2_rn(re.re, p2neg(im.im)), __fadd2_rn(re.im, im.re)};
    });
    sfor<0, N>([&](auto ic) { a[decltype(ic)::value] = out[decltype(ic)::value]; });
  } else {
    constexpr int P = first_radix<N>();
    constexpr int Q = N / P;
    static_assert(P * Q == N && P > 1 && Q > 1, "unsupported DFT size");
    PairC b[N];
    sfor<0, Q>([&](auto n2c) {
      constexpr int n2 = decltype(n2c)::value;
      PairC t[P];
      sfor<0, P>([&](auto n1c) { t[decltype(n1c)::value] = a[Q * decltype(n1c)::value + n2]; });
      pair_dft<P>(t);
      sfor<0, P>([&](auto k1c) {
        constexpr int k1 = decltype(k1c)::value;
        b[k1 * Q + n2] = pc_twc<N, n2 * k1>(t[k1]);
      });
    });
    sfor<0, P>([&](auto k1c) {
      constexpr int k1 = decltype(k1c)::value;
      pair_dft<Q>(&b[k1 * Q]);
      sfor<0, Q>([&](auto k2c) { a[k1 + P * decltype(k2c)::value] = b[k1 * Q + decltype(k2c)::value]; });
    });
  }
}

}  // namespace gbn
