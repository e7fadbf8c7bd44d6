// aw_common.cuh — shared device helpers for the sm_100a registration kernels.
//
// Interpolation arithmetic follows the reference CPU routines operation by
// operation (HField3DUtils::trilerp, Array3DUtils::trilerp,
// HField3DUtils::forwardApply): float positions and data, double weights and
// sums. Every product and sum below is an explicit round-to-nearest
// intrinsic so the compiler cannot contract it into a fused multiply-add;
// with identical inputs the results are bit-identical to the reference.
#pragma once

#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include <utility>

#define AW_HD __host__ __device__ __forceinline__
#define AW_D __device__ __forceinline__

namespace aw {

// HField3DUtils::VectorBackgroundStrategy (UtilitiesDataTypes/HField3DUtils.h:44-49)
enum BgStrategy { BG_PARTIAL_ID = 0, BG_ID = 1, BG_PARTIAL_ZERO = 2, BG_ZERO = 3, BG_CLAMP = 4, BG_WRAP = 5 };

struct Dims {
  int nx, ny, nz;
  AW_HD long n() const { return (long)nx * ny * nz; }
  AW_HD long idx(int x, int y, int z) const { return ((long)z * ny + y) * nx + x; }
};

struct Spacing {
  double x, y, z;
};

// Elementwise launch shape: 128 threads along x, one grid row per (y, z), so
// a thread finds its voxel without any integer division.
constexpr int kRowThreads = 128;
inline dim3 row_grid(const Dims &d) {
  return dim3((unsigned)((d.nx + kRowThreads - 1) / kRowThreads), (unsigned)d.ny, (unsigned)d.nz);
}
struct Voxel {
  int x, y, z;
  long i;
};
AW_D bool voxel_of(const Dims &d, Voxel &v) {
  v.x = blockIdx.x * kRowThreads + threadIdx.x;
  v.y = blockIdx.y;
  v.z = blockIdx.z;
  v.i = ((long)v.z * d.ny + v.y) * d.nx + v.x;
  return v.x < d.nx;
}

// Programmatic dependent launch: a kernel launched by launch_early may begin
// while the kernel before it on the stream is still running, once every block
// of that one has called dependents_may_start (or has ended). It fetches its
// constant tables and sets up its barriers, then waits in
// wait_for_predecessors, before the first access to anything an earlier
// kernel writes or reads, until that kernel has completed. Both calls do
// nothing in a kernel launched in the ordinary way.
AW_D void wait_for_predecessors() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
AW_D void dependents_may_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
// for a kernel with nothing to do before its data is there: its launch alone
// overlaps the end of the kernel before it. None of these calls
// dependents_may_start: with it an LDMM iteration at 128^3 took 3259 us
// against 3105 without and 3135 launched in the ordinary way (the waiting
// blocks take the places of the running kernel's), and an adjoint-shooting
// iteration, which is not replayed from a graph, 4218 without and 4577 in the
// ordinary way.
AW_D void early_entry() { wait_for_predecessors(); }
template <class... P, class... A>
cudaError_t launch_early(void (*kernel)(P...), dim3 grid, unsigned threads, size_t smem,
                         cudaStream_t s, A &&...args) {
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cfg.attrs = &attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, std::forward<A>(args)...);
}

// the outcome of a launch_early, without leaving it behind for the next
// caller of cudaGetLastError
inline cudaError_t launched(cudaError_t e) {
  const cudaError_t last = cudaGetLastError();
  return e != cudaSuccess ? e : last;
}

// n / d for 0 <= n < 2^31 by multiply and shift (round-up method)
struct IdxDiv {
  uint32_t d, mul, l;
  AW_D int div(int n) const { return (int)((__umulhi((uint32_t)n, mul) + (uint32_t)n) >> l); }
};
inline IdxDiv make_idxdiv(uint32_t d) {
  uint32_t l = 0;
  while ((1ull << l) < d) ++l;
  return IdxDiv{d, (uint32_t)(((1ull << 32) * ((1ull << l) - d)) / d + 1), l};
}

// ---- exact-rounding arithmetic -------------------------------------------
AW_D double dmul(double a, double b) { return __dmul_rn(a, b); }
AW_D double dadd(double a, double b) { return __dadd_rn(a, b); }
AW_D double dsub(double a, double b) { return __dsub_rn(a, b); }
AW_D float fmul(float a, float b) { return __fmul_rn(a, b); }
AW_D float fadd(float a, float b) { return __fadd_rn(a, b); }
AW_D float fsub(float a, float b) { return __fsub_rn(a, b); }
AW_D float fdiv(float a, float b) { return __fdiv_rn(a, b); }

// x / d as the reference divides (IEEE, round to nearest). When d is a power
// of two the quotient is x scaled by an exact power of two, and x * (1/d)
// is the same number: the multiply replaces the division sequence.
// A float x divided in double and rounded to float is also one float
// operation where the divisor allows it (div_float): x / d in float when d is
// a float (the double quotient of two floats never rounds onto a float
// midpoint it was not on: 53 >= 2 * 24 + 2, Figueroa 1995), x * (1/d) when d
// is a power of two whose reciprocal is a normal float.
struct DivD {
  double d, r;
  int p2;
  int as;        // div_float: 2 multiply by fr, 1 divide by fd, 0 in double
  float fd, fr;
};
struct DivF {
  float d, r;
  int p2;
};
inline bool host_is_pow2(double d) {
  if (!(d > 0.0)) return false;
  int e = 0;
  const double m = frexp(d, &e);
  return m == 0.5 && e > -1000 && e < 1000;
}
inline DivD make_div(double d) {
  DivD q{d, 1.0 / d, host_is_pow2(d) ? 1 : 0, 0, (float)d, (float)(1.0 / d)};
  if (q.p2 && q.r >= 0x1p-100 && q.r <= 0x1p+100)
    q.as = 2;
  else if ((double)q.fd == d && d >= 0x1p-100 && d <= 0x1p+100)
    q.as = 1;
  return q;
}
inline DivF make_divf(float d) { return DivF{d, 1.0f / d, host_is_pow2((double)d) ? 1 : 0}; }
AW_D double ddiv(double x, const DivD &q) { return q.p2 ? dmul(x, q.r) : __ddiv_rn(x, q.d); }
AW_D float div_float(float x, const DivD &q) {
  if (q.as == 2) return fmul(x, q.fr);
  if (q.as == 1) return fdiv(x, q.fd);
  return __double2float_rn(ddiv((double)x, q));
}
AW_D float fdivq(float x, const DivF &q) { return q.p2 ? fmul(x, q.r) : fdiv(x, q.d); }

// Atlas subjects on grids of their own: a deformation lives on the template
// grid (n voxels per axis) and points into the subject's grid (m voxels per
// axis) through the map of voxel centres of equal physical extent,
// p -> (p + 0.5) * (m / n) - 0.5, in double. `on` is 0 when m == n, and the
// sample point is then h itself, as in the reference's equal-grid atlas.
struct AtlasMap {
  int on;
  double r[3];  // m / n per axis
};
AW_D void atlas_point(const AtlasMap &a, double &x, double &y, double &z) {
  x = dsub(dmul(dadd(x, 0.5), a.r[0]), 0.5);
  y = dsub(dmul(dadd(y, 0.5), a.r[1]), 0.5);
  z = dsub(dmul(dadd(z, 0.5), a.r[2]), 0.5);
}

// floor as the reference computes it: truncate, then step down for
// negative non-integers (Array3DUtils.txx:70-75)
// Positions are clamped to [-2^30, 2^30] first (NaN to -2^30): the same
// floor for every position a grid can hold, and for huge, infinite or NaN
// positions a cell far outside every grid, so fx + 1 cannot overflow and
// the callers' inside/outside tests never pass an out-of-range corner.
AW_D int ref_floor_d(double x) {
  x = fmin(fmax(x, -0x1p30), 0x1p30);
  int f = __double2int_rz(x);
  if (x < 0.0 && x != (double)f) --f;
  return f;
}
AW_D int ref_floor_f(float x) {
  x = fminf(fmaxf(x, -0x1p30f), 0x1p30f);
  int f = __float2int_rz(x);
  if (x < 0.0f && x != __int2float_rn(f)) --f;
  return f;
}

// The cell of a position and its float corner, as ref_floor_f finds them,
// without the conversion unit, which the interpolation kernels' 24 float to
// double conversions a voxel keep half busy: adding 1.5 * 2^23 rounds to the
// nearest integer in the mantissa's low bits, and a value it rounded up steps
// back down. For positions within 2^21 of zero; others (huge, infinite, NaN)
// take ref_floor_f.
AW_D void floor_near(float x, int &i, float &f) {
  const float t = fadd(x, 12582912.0f);
  f = fsub(t, 12582912.0f);
  i = __float_as_int(t) - 0x4b400000;
  if (f > x) {
    f = fsub(f, 1.0f);
    --i;
  }
}
AW_D void cell_of(float x, float y, float z, int &fx, int &fy, int &fz, float &gx, float &gy,
                  float &gz) {
  if (fadd(fadd(fabsf(x), fabsf(y)), fabsf(z)) < 2097152.0f) {
    floor_near(x, fx, gx);
    floor_near(y, fy, gy);
    floor_near(z, fz, gz);
  } else {
    fx = ref_floor_f(x);
    fy = ref_floor_f(y);
    fz = ref_floor_f(z);
    gx = __int2float_rn(fx);
    gy = __int2float_rn(fy);
    gz = __int2float_rn(fz);
  }
}

// ((omt*(omu*(c0*omv + c7*v) + u*(c3*omv + c4*v))) + t*(omu*(c1*omv + c6*v) + u*(c2*omv + c5*v)))
AW_D double lerp_tree(const float c[8], double t, double u, double v, double omt, double omu,
                      double omv) {
  const double a = dmul(omt, dadd(dmul(omu, dadd(dmul((double)c[0], omv), dmul((double)c[7], v))),
                                  dmul(u, dadd(dmul((double)c[3], omv), dmul((double)c[4], v)))));
  const double b = dmul(t, dadd(dmul(omu, dadd(dmul((double)c[1], omv), dmul((double)c[6], v))),
                                dmul(u, dadd(dmul((double)c[2], omv), dmul((double)c[5], v)))));
  return dadd(a, b);
}

// The same tree in float with fused multiply-adds, a + t (b - a) per lerp
// (x first, then y, then z): the fast-interpolation mode. Not bit-identical
// to the double tree; the difference is a few float ulps of the result.
AW_D float lerpf(float a, float b, float t) { return fmaf(t, b - a, a); }
AW_D float lerp_tree_f(const float c[8], float t, float u, float v) {
  const float x00 = lerpf(c[0], c[1], t), x10 = lerpf(c[3], c[2], t);
  const float x01 = lerpf(c[7], c[6], t), x11 = lerpf(c[4], c[5], t);
  return lerpf(lerpf(x00, x10, u), lerpf(x01, x11, u), v);
}

// Scalar trilinear sample, background value per out-of-volume corner
// (Array3DUtils::trilerp<T, BACKGROUND_STRATEGY_VAL>, Array3DUtils.txx:59-232).
// FAST: the float tree (lerp_tree_f) on float fractions.
template <bool FAST = false>
AW_D float trilerp_scalar(const float *__restrict__ a, const Dims d, double x, double y, double z,
                          float bg) {
  const int fx = ref_floor_d(x), fy = ref_floor_d(y), fz = ref_floor_d(z);
  const int cx = fx + 1, cy = fy + 1, cz = fz + 1;
  const double t = dsub(x, (double)fx), u = dsub(y, (double)fy), v = dsub(z, (double)fz);
  const double omt = FAST ? 0.0 : dsub(1.0, t), omu = FAST ? 0.0 : dsub(1.0, u),
               omv = FAST ? 0.0 : dsub(1.0, v);
  float c[8];
  const bool inside = fx >= 0 && cx < d.nx && fy >= 0 && cy < d.ny && fz >= 0 && cz < d.nz;
  if (inside) {
    // 32-bit offsets: every grid here has fewer than 2^31 voxels
    const int b = (fz * d.ny + fy) * d.nx + fx;
    const int sy = d.nx, sz = d.nx * d.ny;
    c[0] = __ldg(a + b);
    c[1] = __ldg(a + b + 1);
    c[2] = __ldg(a + b + sy + 1);
    c[3] = __ldg(a + b + sy);
    c[4] = __ldg(a + b + sy + sz);
    c[5] = __ldg(a + b + sy + sz + 1);
    c[6] = __ldg(a + b + sz + 1);
    c[7] = __ldg(a + b + sz);
  } else {
    const bool fxi = fx >= 0 && fx < d.nx, fyi = fy >= 0 && fy < d.ny, fzi = fz >= 0 && fz < d.nz;
    const bool cxi = cx >= 0 && cx < d.nx, cyi = cy >= 0 && cy < d.ny, czi = cz >= 0 && cz < d.nz;
    c[0] = (fxi && fyi && fzi) ? __ldg(a + d.idx(fx, fy, fz)) : bg;
    c[1] = (cxi && fyi && fzi) ? __ldg(a + d.idx(cx, fy, fz)) : bg;
    c[2] = (cxi && cyi && fzi) ? __ldg(a + d.idx(cx, cy, fz)) : bg;
    c[3] = (fxi && cyi && fzi) ? __ldg(a + d.idx(fx, cy, fz)) : bg;
    c[4] = (fxi && cyi && czi) ? __ldg(a + d.idx(fx, cy, cz)) : bg;
    c[5] = (cxi && cyi && czi) ? __ldg(a + d.idx(cx, cy, cz)) : bg;
    c[6] = (cxi && fyi && czi) ? __ldg(a + d.idx(cx, fy, cz)) : bg;
    c[7] = (fxi && fyi && czi) ? __ldg(a + d.idx(fx, fy, cz)) : bg;
  }
  if (FAST) return lerp_tree_f(c, (float)t, (float)u, (float)v);
  return __double2float_rn(lerp_tree(c, t, u, v, omt, omu, omv));
}

// The eight corners of a cell on a grid: clamped offsets, and which corners
// lie inside.
struct CellCorners {
  int x[2], y[2], z[2];      // offsets along each axis
  bool ix[2], iy[2], iz[2];
  AW_D int at(int c) const { return z[kZ(c)] + y[kY(c)] + x[kX(c)]; }
  AW_D bool in(int c) const { return ix[kX(c)] && iy[kY(c)] && iz[kZ(c)]; }
  // corner c of the reference's order is (x, y, z) = (kX, kY, kZ)
  AW_D static constexpr int kX(int c) { return (0x66 >> c) & 1; }
  AW_D static constexpr int kY(int c) { return (0x3c >> c) & 1; }
  AW_D static constexpr int kZ(int c) { return (0xf0 >> c) & 1; }
};
AW_D CellCorners cell_corners(const Dims &d, int fx, int fy, int fz) {
  CellCorners k;
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    k.x[i] = min(max(fx + i, 0), d.nx - 1);
    k.y[i] = min(max(fy + i, 0), d.ny - 1) * d.nx;
    k.z[i] = min(max(fz + i, 0), d.nz - 1) * (d.nx * d.ny);
    k.ix[i] = (unsigned)(fx + i) < (unsigned)d.nx;
    k.iy[i] = (unsigned)(fy + i) < (unsigned)d.ny;
    k.iz[i] = (unsigned)(fz + i) < (unsigned)d.nz;
  }
  return k;
}
AW_D bool cell_inside(const Dims &d, int fx, int fy, int fz) {
  return (unsigned)fx < (unsigned)(d.nx - 1) && (unsigned)fy < (unsigned)(d.ny - 1) &&
         (unsigned)fz < (unsigned)(d.nz - 1);
}
// whether any of the warp's threads here has p: kernels whose common case
// and border case differ choose one for the whole warp, so that a warp with
// a single border voxel does not run both, one after the other
AW_D bool warp_any(bool p) { return __any_sync(__activemask(), p); }

// The same at a float position. A cell inside the volume has no negative
// coordinate, and x - floor(x) of a float x >= 0 is a float: there the
// fractions are formed in float and widened. A warp with a cell at the
// border fetches clamped corners and selects.
template <bool FAST = false>
AW_D float trilerp_scalar(const float *__restrict__ a, const Dims d, float x, float y, float z,
                          float bg) {
  int fx, fy, fz;
  float gx, gy, gz;
  cell_of(x, y, z, fx, fy, fz, gx, gy, gz);
  float c[8];
  double t, u, v;
  if (!warp_any(!cell_inside(d, fx, fy, fz))) {
    const int b = (fz * d.ny + fy) * d.nx + fx;
    const int sy = d.nx, sz = d.nx * d.ny;
    c[0] = __ldg(a + b);
    c[1] = __ldg(a + b + 1);
    c[2] = __ldg(a + b + sy + 1);
    c[3] = __ldg(a + b + sy);
    c[4] = __ldg(a + b + sy + sz);
    c[5] = __ldg(a + b + sy + sz + 1);
    c[6] = __ldg(a + b + sz + 1);
    c[7] = __ldg(a + b + sz);
    t = (double)fsub(x, gx);
    u = (double)fsub(y, gy);
    v = (double)fsub(z, gz);
  } else {
    const CellCorners k = cell_corners(d, fx, fy, fz);
#pragma unroll
    for (int i = 0; i < 8; ++i) c[i] = __ldg(a + k.at(i));
#pragma unroll
    for (int i = 0; i < 8; ++i) c[i] = k.in(i) ? c[i] : bg;
    t = dsub((double)x, (double)gx);
    u = dsub((double)y, (double)gy);
    v = dsub((double)z, (double)gz);
  }
  if (FAST) return lerp_tree_f(c, (float)t, (float)u, (float)v);
  return __double2float_rn(lerp_tree(c, t, u, v, dsub(1.0, t), dsub(1.0, u), dsub(1.0, v)));
}

AW_D int safe_mod(int r, int m) {
  r %= m;
  return r < 0 ? r + m : r;
}

// Vector trilinear sample with the reference's background strategies
// (HField3DUtils::trilerp, HField3DUtils.txx:1972-2300). Position in float,
// fractional part formed in float, weights and sums in double. `scale`
// multiplies each fetched corner value in float first (it reproduces
// interpolating a field that the reference scaled in place beforehand);
// pass 1.0f for none. FAST: the float tree (lerp_tree_f).
template <bool FAST = false>
AW_D void trilerp_vector(const float *__restrict__ hx, const float *__restrict__ hy,
                         const float *__restrict__ hz, const Dims d, float x, float y, float z,
                         int bgs, float scale, float &ox, float &oy, float &oz) {
  int fx, fy, fz;
  float gx, gy, gz;
  cell_of(x, y, z, fx, fy, fz, gx, gy, gz);
  const float tf = fsub(x, gx), uf = fsub(y, gy), vf = fsub(z, gz);
  const double t = (double)tf, u = (double)uf, v = (double)vf;
  const double omt = FAST ? 0.0 : dsub(1.0, t), omu = FAST ? 0.0 : dsub(1.0, u),
               omv = FAST ? 0.0 : dsub(1.0, v);
  float cxv[8], cyv[8], czv[8];
  if (bgs == BG_WRAP || bgs == BG_CLAMP) {
    int cx = fx + 1, cy = fy + 1, cz = fz + 1;
    if (bgs == BG_WRAP) {
      fx = safe_mod(fx, d.nx); fy = safe_mod(fy, d.ny); fz = safe_mod(fz, d.nz);
      cx = safe_mod(cx, d.nx); cy = safe_mod(cy, d.ny); cz = safe_mod(cz, d.nz);
    } else {
      if (fx < 0) { fx = 0; if (cx < 0) cx = 0; }
      if (cx >= d.nx) { cx = d.nx - 1; if (fx >= d.nx) fx = d.nx - 1; }
      if (fy < 0) { fy = 0; if (cy < 0) cy = 0; }
      if (cy >= d.ny) { cy = d.ny - 1; if (fy >= d.ny) fy = d.ny - 1; }
      if (fz < 0) { fz = 0; if (cz < 0) cz = 0; }
      if (cz >= d.nz) { cz = d.nz - 1; if (fz >= d.nz) fz = d.nz - 1; }
    }
    const int X[2] = {fx, cx}, Y[2] = {fy, cy}, Z[2] = {fz, cz};
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      const int i = (Z[CellCorners::kZ(c)] * d.ny + Y[CellCorners::kY(c)]) * d.nx +
                    X[CellCorners::kX(c)];
      cxv[c] = __ldg(hx + i);
      cyv[c] = __ldg(hy + i);
      czv[c] = __ldg(hz + i);
    }
    if (scale != 1.0f) {
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        cxv[c] = fmul(cxv[c], scale);
        cyv[c] = fmul(cyv[c], scale);
        czv[c] = fmul(czv[c], scale);
      }
    }
  } else {
    const bool inside = cell_inside(d, fx, fy, fz);
    if (!inside && (bgs == BG_ID || bgs == BG_ZERO)) {
      ox = bgs == BG_ID ? x : 0.f;
      oy = bgs == BG_ID ? y : 0.f;
      oz = bgs == BG_ID ? z : 0.f;
      return;
    }
    if (!warp_any(!inside)) {
      const int b = (fz * d.ny + fy) * d.nx + fx;
      const int sy = d.nx, sz = d.nx * d.ny;
      const int off[8] = {b, b + 1, b + sy + 1, b + sy, b + sy + sz, b + sy + sz + 1, b + sz + 1,
                          b + sz};
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        cxv[c] = __ldg(hx + off[c]);
        cyv[c] = __ldg(hy + off[c]);
        czv[c] = __ldg(hz + off[c]);
      }
      if (scale != 1.0f) {
#pragma unroll
        for (int c = 0; c < 8; ++c) {
          cxv[c] = fmul(cxv[c], scale);
          cyv[c] = fmul(cyv[c], scale);
          czv[c] = fmul(czv[c], scale);
        }
      }
    } else {
      // a border cell in the warp: clamped corners, and outside the volume
      // the corner's own place (PARTIAL_ID) or zero
      const CellCorners k = cell_corners(d, fx, fy, fz);
      const bool pid = bgs == BG_PARTIAL_ID;
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        const int i = k.at(c);
        cxv[c] = fmul(__ldg(hx + i), scale);
        cyv[c] = fmul(__ldg(hy + i), scale);
        czv[c] = fmul(__ldg(hz + i), scale);
      }
      const float X[2] = {gx, __int2float_rn(fx + 1)}, Y[2] = {gy, __int2float_rn(fy + 1)},
                  Z[2] = {gz, __int2float_rn(fz + 1)};
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        const bool in = k.in(c);
        cxv[c] = in ? cxv[c] : (pid ? X[CellCorners::kX(c)] : 0.f);
        cyv[c] = in ? cyv[c] : (pid ? Y[CellCorners::kY(c)] : 0.f);
        czv[c] = in ? czv[c] : (pid ? Z[CellCorners::kZ(c)] : 0.f);
      }
    }
  }
  if (FAST) {
    ox = lerp_tree_f(cxv, tf, uf, vf);
    oy = lerp_tree_f(cyv, tf, uf, vf);
    oz = lerp_tree_f(czv, tf, uf, vf);
    return;
  }
  ox = __double2float_rn(lerp_tree(cxv, t, u, v, omt, omu, omv));
  oy = __double2float_rn(lerp_tree(cyv, t, u, v, omt, omu, omv));
  oz = __double2float_rn(lerp_tree(czv, t, u, v, omt, omu, omv));
}

// ---- warp reductions --------------------------------------------------------
AW_D double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  return v;
}
AW_D float warp_max(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_down_sync(0xffffffffu, v, o));
  return v;
}

}  // namespace aw
