// Register DFTs of any radix up to 16, and the small arithmetic the transform kernels share.
//
// The in-place shared-memory transforms for any line length are in kwb_generic.cu, the
// register-resident ones for the lengths they cover in kwb_fast_impl.cuh.
#pragma once
#include <type_traits>

#include "kwb_internal.h"

namespace kwb {

__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
  return make_float2(fmaf(a.x, b.x, -a.y * b.y), fmaf(a.x, b.y, a.y * b.x));
}
// (packed FP32 pairs: per component the round-to-nearest result of the scalar operation, in one
// instruction for both)
__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return __fadd2_rn(a, make_float2(-b.x, -b.y)); }
__device__ __forceinline__ float2 cscale(float2 a, float s) { return __fmul2_rn(a, make_float2(s, s)); }
__device__ __forceinline__ float2 cfma(float s, float2 a, float2 b) { return __ffma2_rn(make_float2(s, s), a, b); }
// multiply by -i (forward) or +i (inverse)
template <bool INV>
__device__ __forceinline__ float2 mul_mi(float2 a) {
  return INV ? make_float2(-a.y, a.x) : make_float2(a.y, -a.x);
}

template <int R, bool INV>
struct Dft;

template <bool INV>
struct Dft<2, INV> {
  __device__ __forceinline__ static void run(float2 (&v)[2]) {
    float2 a = cadd(v[0], v[1]);
    float2 b = csub(v[0], v[1]);
    v[0] = a;
    v[1] = b;
  }
};

template <bool INV>
struct Dft<4, INV> {
  __device__ __forceinline__ static void run(float2 (&v)[4]) {
    float2 t0 = cadd(v[0], v[2]), t1 = csub(v[0], v[2]);
    float2 t2 = cadd(v[1], v[3]), t3 = mul_mi<INV>(csub(v[1], v[3]));
    v[0] = cadd(t0, t2);
    v[2] = csub(t0, t2);
    v[1] = cadd(t1, t3);
    v[3] = csub(t1, t3);
  }
};

// ---- register DFTs of any radix up to 16

// cos and sin of 2 pi m / R, m < R, in double by their Taylor series after folding into [0, pi/4]
// (evaluated at compile time, rounded once to FP32).
struct CosSin {
  double c, s;
};
__host__ __device__ constexpr CosSin cos_sin_turn(int m, int R) {
  // m/R of a turn; fold by symmetry to the first octant, in integers (eighths of a turn: 8 m / R)
  bool neg_s = false, neg_c = false, swap = false;
  if (2 * m > R) {
    m = R - m;
    neg_s = true;
  }
  // now 0 <= m/R <= 1/2
  int num = m, den = R;  // angle = num/den turns
  if (4 * num > den) {   // second quadrant: pi - x
    num = den - 2 * num;
    den = 2 * den;
    neg_c = true;
  }
  if (8 * num > den) {  // beyond pi/4: pi/2 - x
    num = den - 4 * num;
    den = 4 * den;
    swap = true;
  }
  const double x = 6.283185307179586476925286766559 * num / den;
  double c = 0.0, s = 0.0, t = 1.0;
  for (int k = 0; k < 24; ++k) {
    const double v = ((k / 2) % 2 == 0) ? t : -t;
    if (k % 2 == 0) c += v;
    else s += v;
    t = t * x / (k + 1);
  }
  const double cc = swap ? s : c, ss = swap ? c : s;
  return CosSin{neg_c ? -cc : cc, neg_s ? -ss : ss};
}
// (value and the remainder of its rounding to FP32: the constants of a radix act on every butterfly
// alike, so an error in one is a gain, the same on every step, that adds up over a simulation --
// 5e-8 a convolution at N = 100, 1e-5 over 200 steps -- where the roundings of the arithmetic average
// out)
template <int R>
struct Roots {
  float c[R], s[R], cl[R], sl[R];
};
template <int R>
__host__ __device__ constexpr Roots<R> make_roots() {
  Roots<R> r{};
  for (int m = 0; m < R; ++m) {
    const CosSin v = cos_sin_turn(m, R);
    r.c[m] = (float)v.c;
    r.s[m] = (float)v.s;
    r.cl[m] = (float)(v.c - (double)r.c[m]);
    r.sl[m] = (float)(v.s - (double)r.s[m]);
  }
  return r;
}

// v exp(-+ 2 pi i m / R) for a compile-time m
template <int R, bool INV>
__device__ __forceinline__ float2 root_mul(float2 v, int m) {
  constexpr Roots<R> W = make_roots<R>();
  m %= R;
  if (m == 0) return v;
  if (4 * m == R) return mul_mi<INV>(v);
  if (2 * m == R) return make_float2(-v.x, -v.y);
  if (4 * m == 3 * R) return mul_mi<!INV>(v);
  const float c = W.c[m], s = INV ? -W.s[m] : W.s[m];
  const float cl = W.cl[m], sl = INV ? -W.sl[m] : W.sl[m];
  return make_float2(fmaf(v.x, c, fmaf(v.y, s, fmaf(v.x, cl, v.y * sl))),
                     fmaf(v.y, c, fmaf(-v.x, s, fmaf(v.y, cl, -v.x * sl))));
}

__host__ __device__ constexpr int first_factor(int R) {
  return R % 4 == 0 && R > 4 ? 4 : R % 3 == 0 && R > 3 ? 3 : R % 2 == 0 && R > 2 ? 2 : R;
}
// R-point DFT in registers, natural order in and out: R = 1, 2, 4, an odd prime (pairs v_j +-
// v_{R-j}), or one Cooley-Tukey step P * Q (n = Q n1 + n2, k = k1 + P k2).
template <int R, bool INV>
__device__ __forceinline__ void dft_any(float2 (&v)[R]) {
  constexpr int P = first_factor(R);
  if constexpr (R == 1) {
    return;
  } else if constexpr (R == 2 || R == 4) {
    Dft<R, INV>::run(v);
  } else if constexpr (P == R) {
    constexpr Roots<R> W = make_roots<R>();
    constexpr int H = (R - 1) / 2;
    float2 t[H], d[H];
    float2 sum = v[0];
    const float2 x0 = v[0];
#pragma unroll
    for (int j = 0; j < H; ++j) {
      t[j] = cadd(v[j + 1], v[R - 1 - j]);
      d[j] = csub(v[j + 1], v[R - 1 - j]);
      sum = cadd(sum, t[j]);
    }
    v[0] = sum;
#pragma unroll
    for (int k = 1; k <= H; ++k) {
      float2 a = make_float2(0.f, 0.f), b = a;
#pragma unroll
      for (int j = 1; j <= H; ++j) {  // the remainders first: the small terms
        const float c = W.cl[(j * k) % R], s = W.sl[(j * k) % R];
        a = cfma(c, t[j - 1], a);
        b = cfma(s, d[j - 1], b);
      }
#pragma unroll
      for (int j = 1; j <= H; ++j) {
        const float c = W.c[(j * k) % R], s = W.s[(j * k) % R];
        a = cfma(c, t[j - 1], a);
        b = cfma(s, d[j - 1], b);
      }
      a = cadd(a, x0);
      b = mul_mi<INV>(b);
      v[k] = cadd(a, b);
      v[R - k] = csub(a, b);
    }
  } else {
    constexpr int Q = R / P;
    float2 a[R];
#pragma unroll
    for (int n2 = 0; n2 < Q; ++n2) {
      float2 w[P];
#pragma unroll
      for (int n1 = 0; n1 < P; ++n1) w[n1] = v[Q * n1 + n2];
      dft_any<P, INV>(w);
#pragma unroll
      for (int k1 = 0; k1 < P; ++k1) a[n2 * P + k1] = root_mul<R, INV>(w[k1], n2 * k1);
    }
#pragma unroll
    for (int k1 = 0; k1 < P; ++k1) {
      float2 w[Q];
#pragma unroll
      for (int n2 = 0; n2 < Q; ++n2) w[n2] = a[n2 * P + k1];
      dft_any<Q, INV>(w);
#pragma unroll
      for (int k2 = 0; k2 < Q; ++k2) v[k1 + P * k2] = w[k2];
    }
  }
}

__device__ __forceinline__ int fdiv(int n, FastDiv d) {
  return (int)((__umulhi((unsigned)n, d.mul) + (unsigned)n) >> d.shift);
}

}  // namespace kwb
