// fft_smem.cuh — complex arithmetic and small butterflies shared by the
// transforms. Twiddles W_n^m = exp(-2*pi*i*m/n) are computed on the host in
// double and rounded to float once. Forward is sign -1, inverse +1; both
// unnormalised, as FFTW/cuFFT.
#pragma once

#include "aw_common.cuh"

namespace aw {

struct FFTAxis {
  const float2 *tw;  // n entries, W_n^m (forward sign)
};

AW_D float2 cmul(float2 a, float2 b) {
  return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
AW_D float2 cadd(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
AW_D float2 csub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
// multiply by sign*i
template <int SIGN>
AW_D float2 mul_si(float2 a) {
  return SIGN < 0 ? make_float2(a.y, -a.x) : make_float2(-a.y, a.x);
}

template <int SIGN>
AW_D float2 twiddle(const float2 *__restrict__ tw, int m) {
  const float2 w = __ldg(tw + m);
  return SIGN < 0 ? w : make_float2(w.x, -w.y);
}

template <int SIGN>
AW_D void bfly4(float2 *v) {
  const float2 s02 = cadd(v[0], v[2]), d02 = csub(v[0], v[2]);
  const float2 s13 = cadd(v[1], v[3]), d13 = mul_si<SIGN>(csub(v[1], v[3]));
  v[0] = cadd(s02, s13);
  v[2] = csub(s02, s13);
  v[1] = cadd(d02, d13);
  v[3] = csub(d02, d13);
}

template <int SIGN>
AW_D void bfly8(float2 *v) {
  float2 e[4] = {v[0], v[2], v[4], v[6]};
  float2 o[4] = {v[1], v[3], v[5], v[7]};
  bfly4<SIGN>(e);
  bfly4<SIGN>(o);
  const float r = 0.70710678118654752440f;
  // W8^u for u = 1, 2, 3 with the transform's sign
  const float2 w1 = make_float2(r, SIGN * r);
  const float2 w3 = make_float2(-r, SIGN * r);
  o[1] = cmul(o[1], w1);
  o[2] = mul_si<SIGN>(o[2]);
  o[3] = cmul(o[3], w3);
#pragma unroll
  for (int u = 0; u < 4; ++u) {
    v[u] = cadd(e[u], o[u]);
    v[u + 4] = csub(e[u], o[u]);
  }
}

}  // namespace aw
