// fr_fft.cuh -- discrete Fourier transforms of a few points in registers, for
// the transforms built on them (fr_slice.cu, fr_lines.cu).
#pragma once
#include <cuda_runtime.h>

#include <utility>

namespace fr {
namespace fft {

// cos and sin of 2 pi k / R by their Taylor series on an angle of at most pi
constexpr double kTwoPi = 6.283185307179586476925286766559;
constexpr double turn(int k, int R) {
  const int m = ((k % R) + R) % R;
  return kTwoPi * (2 * m > R ? m - R : m) / R;
}
constexpr double ccos(double x) {
  double t = 1.0, s = 1.0;
  for (int i = 1; i < 24; i++) {
    t *= -x * x / ((2.0 * i - 1.0) * (2.0 * i));
    s += t;
  }
  return s;
}
constexpr double csin(double x) {
  double t = x, s = x;
  for (int i = 1; i < 24; i++) {
    t *= -x * x / ((2.0 * i) * (2.0 * i + 1.0));
    s += t;
  }
  return s;
}

template <class F, int... I>
__device__ __forceinline__ void each(std::integer_sequence<int, I...>, F f) {
  (f(std::integral_constant<int, I>{}), ...);
}
template <int N, class F> __device__ __forceinline__ void each(F f) {
  each(std::make_integer_sequence<int, N>{}, f);
}

// Sums and differences of complex values, one packed operation each.
__device__ __forceinline__ float2 cadd(float2 a, float2 b) {
  float2 r;
  asm("{.reg .b64 x, y;\n mov.b64 x, {%2, %3};\n mov.b64 y, {%4, %5};\n"
      " add.rn.f32x2 x, x, y;\n mov.b64 {%0, %1}, x;}"
      : "=f"(r.x), "=f"(r.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return r;
}
__device__ __forceinline__ float2 csub(float2 a, float2 b) {
  return cadd(a, make_float2(-b.x, -b.y));
}
// a * (c + i s), s negated for the forward direction by the caller
__device__ __forceinline__ float2 cmul(float2 a, float c, float s) {
  return make_float2(fmaf(a.x, c, -a.y * s), fmaf(a.x, s, a.y * c));
}

// How a composite radix splits into two.
constexpr int first_factor(int R) {
  return R == 16 || R == 12 || R == 20 || R == 8 || R == 4 ? (R == 4 ? 2 : 4)
         : R % 2 == 0                                      ? 2
         : R % 3 == 0                                      ? 3
                                                           : R;
}

// v <- DFT of v, natural order; DIR = -1 forward (exp(-i..)), +1 inverse.
template <int R, int DIR> __device__ __forceinline__ void dft(float2 (&v)[R]) {
  constexpr int A = first_factor(R), B = R / A;
  if constexpr (R == 2) {
    const float2 a = v[0], b = v[1];
    v[0] = cadd(a, b);
    v[1] = csub(a, b);
  } else if constexpr (R == 4) {
    const float2 a = cadd(v[0], v[2]), b = csub(v[0], v[2]), c = cadd(v[1], v[3]),
                 d = csub(v[1], v[3]);
    const float2 e = make_float2(-DIR * d.y, DIR * d.x);   // (i DIR) d
    v[0] = cadd(a, c);
    v[2] = csub(a, c);
    v[1] = cadd(b, e);
    v[3] = csub(b, e);
  } else if constexpr (B == 1) {
    // odd prime: pairs (n, R-n) as sums and differences
    float2 s[R / 2 + 1], d[R / 2 + 1];
    float2 sum = v[0];
    each<R / 2>([&](auto I) {
      constexpr int n = I.value + 1;
      s[n] = cadd(v[n], v[R - n]);
      d[n] = csub(v[n], v[R - n]);
      sum = cadd(sum, s[n]);
    });
    const float2 v0 = v[0];
    each<R / 2>([&](auto K) {
      constexpr int k = K.value + 1;
      float2 re = v0, im = make_float2(0.f, 0.f);
      each<R / 2>([&](auto I) {
        constexpr int n = I.value + 1;
        constexpr float c = (float)ccos(turn(n * k, R)), q = (float)(DIR * csin(turn(n * k, R)));
        re.x = fmaf(s[n].x, c, re.x);
        re.y = fmaf(s[n].y, c, re.y);
        im.x = fmaf(d[n].y, -q, im.x);   // i q d
        im.y = fmaf(d[n].x, q, im.y);
      });
      v[k] = cadd(re, im);
      v[R - k] = csub(re, im);
    });
    v[0] = sum;
  } else {
    // n = n1 B + n2, k = k1 + A k2
    float2 u[B][A];
    each<B>([&](auto I) {
      constexpr int n2 = I.value;
      float2 t[A];
      each<A>([&](auto J) { t[J.value] = v[J.value * B + n2]; });
      dft<A, DIR>(t);
      each<A>([&](auto J) {
        constexpr int k1 = J.value;
        if constexpr (n2 == 0 || k1 == 0) u[n2][k1] = t[k1];
        else
          u[n2][k1] = cmul(t[k1], (float)ccos(turn(n2 * k1, R)),
                           (float)(DIR * csin(turn(n2 * k1, R))));
      });
    });
    each<A>([&](auto J) {
      constexpr int k1 = J.value;
      float2 t[B];
      each<B>([&](auto I) { t[I.value] = u[I.value][k1]; });
      dft<B, DIR>(t);
      each<B>([&](auto I) { v[k1 + A * I.value] = t[I.value]; });
    });
  }
}

}  // namespace fft
}  // namespace fr
