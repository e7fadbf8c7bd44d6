// dft_reg.cuh — DFTs of a compile-time length held in one thread's
// registers: the butterflies of the in-place line transforms of
// fluid_any.cu. Natural order in and out, unnormalised, SIGN the exponent's.
//
// Lengths up to 16: the primes 2, 3, 5, 7, 11, 13 directly (the odd ones as
// cosine and sine sums over the pairs x[j] +- x[R-j]), the others as two
// steps A x B (Cooley & Tukey 1965) with compile-time twiddles, each rounded
// once from double.
#pragma once

#include <type_traits>

#include "aw_common.cuh"
#include "fft_smem.cuh"

namespace aw {

// cos and sin of 2 pi m / n at compile time: the angle reduced to an eighth
// of the circle, then the Taylor series there (15 terms, below 1e-17)
constexpr double kTwoPi = 6.28318530717958647692528676655900577;
constexpr double series_cos(double x) {
  double t = 1.0, s = 1.0;
  for (int k = 1; k < 16; ++k) {
    t *= -x * x / ((2 * k - 1) * (2 * k));
    s += t;
  }
  return s;
}
constexpr double series_sin(double x) {
  double t = x, s = x;
  for (int k = 1; k < 16; ++k) {
    t *= -x * x / ((2 * k) * (2 * k + 1));
    s += t;
  }
  return s;
}
constexpr double unit_cos(int m, int n) {
  m %= n;
  if (2 * m > n) m = n - m;                              // cos(-a) = cos a
  if (4 * m > n) return -series_cos(kTwoPi * (n - 2 * m) / (2.0 * n));  // cos(pi - a)
  return 8 * m > n ? series_sin(kTwoPi * (n - 4 * m) / (4.0 * n)) : series_cos(kTwoPi * m / n);
}
constexpr double unit_sin(int m, int n) {
  m %= n;
  if (2 * m > n) return -unit_sin(n - m, n);
  if (4 * m > n) return unit_sin(n - 2 * m, 2 * n);      // sin(pi - a), a = 2 pi m / n
  return 8 * m > n ? series_cos(kTwoPi * (n - 4 * m) / (4.0 * n)) : series_sin(kTwoPi * m / n);
}

template <int I, int N, class F>
AW_D void static_for(const F &f) {
  if constexpr (I < N) {
    f(std::integral_constant<int, I>());
    static_for<I + 1, N>(f);
  }
}

// a * exp(SIGN 2 pi i M / R)
template <int SIGN, int M, int R>
AW_D float2 mul_unit(float2 a) {
  constexpr int m = M % R;
  if constexpr (m == 0) {
    return a;
  } else if constexpr (4 * m == R) {
    return mul_si<SIGN>(a);
  } else if constexpr (2 * m == R) {
    return make_float2(-a.x, -a.y);
  } else if constexpr (4 * m == 3 * R) {
    return mul_si<-SIGN>(a);
  } else {
    constexpr float c = (float)unit_cos(m, R), s = (float)(SIGN * unit_sin(m, R));
    return make_float2(a.x * c - a.y * s, a.x * s + a.y * c);
  }
}

// first factor of the two-step split of R (1: a prime, done directly)
constexpr int dft_split(int R) {
  return R % 4 == 0 && R > 4 ? 4 : (R == 4 || (R % 2 == 0 && R > 2)) ? 2 : R % 3 == 0 && R > 3 ? 3 : 1;
}

template <int SIGN, int R>
AW_D void dft(float2 (&v)[R]) {
  constexpr int A = dft_split(R);
  if constexpr (R == 1) {
  } else if constexpr (R == 2) {
    const float2 a = v[0], b = v[1];
    v[0] = cadd(a, b);
    v[1] = csub(a, b);
  } else if constexpr (A == 1) {
    // an odd prime: y[k], y[R-k] = x0 + sum cos t_j  +- SIGN i sum sin u_j
    constexpr int H = (R - 1) / 2;
    float2 t[H], u[H];
    float2 s = v[0];
#pragma unroll
    for (int j = 0; j < H; ++j) {
      t[j] = cadd(v[1 + j], v[R - 1 - j]);
      u[j] = csub(v[1 + j], v[R - 1 - j]);
      s = cadd(s, t[j]);
    }
    const float2 x0 = v[0];
    v[0] = s;
    static_for<1, H + 1>([&](auto kc) {
      constexpr int k = decltype(kc)::value;
      float2 a = x0, b = make_float2(0.f, 0.f);
      static_for<1, H + 1>([&](auto jc) {
        constexpr int j = decltype(jc)::value;
        constexpr float c = (float)unit_cos(j * k, R), sn = (float)(SIGN * unit_sin(j * k, R));
        a.x = fmaf(c, t[j - 1].x, a.x);
        a.y = fmaf(c, t[j - 1].y, a.y);
        b.x = j == 1 ? sn * u[0].x : fmaf(sn, u[j - 1].x, b.x);
        b.y = j == 1 ? sn * u[0].y : fmaf(sn, u[j - 1].y, b.y);
      });
      v[k] = make_float2(a.x - b.y, a.y + b.x);
      v[R - k] = make_float2(a.x + b.y, a.y - b.x);
    });
  } else {
    constexpr int B = R / A;
    // elements a * B + b: DFT over a, twiddle, DFT over b; X[ka + A kb]
    float2 w[A][B];
    static_for<0, B>([&](auto bc) {
      constexpr int b = decltype(bc)::value;
      float2 x[A];
#pragma unroll
      for (int a = 0; a < A; ++a) x[a] = v[a * B + b];
      dft<SIGN, A>(x);
      static_for<0, A>([&](auto ac) {
        constexpr int a = decltype(ac)::value;
        w[a][b] = mul_unit<SIGN, a * b, R>(x[a]);
      });
    });
#pragma unroll
    for (int a = 0; a < A; ++a) {
      dft<SIGN, B>(w[a]);
#pragma unroll
      for (int b = 0; b < B; ++b) v[a + A * b] = w[a][b];
    }
  }
}

}  // namespace aw
