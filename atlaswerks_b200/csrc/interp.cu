// interp.cu — trilinear apply / compose / gradient kernels and the greedy
// force-side and update-side kernels that use them.
//
// One thread per output voxel, consecutive threads on consecutive x, so the
// streamed planes (h, v, I1, outputs) are read and written fully coalesced;
// the gathers (I0 at h(x), h at x + v) hit L1/L2 because displacements are
// small. Arithmetic follows the reference CPU routines exactly (see
// aw_common.cuh), so with identical inputs the outputs are bit-identical.
#include "interp.cuh"

namespace aw {

namespace {

constexpr int kThreads = kRowThreads;

// HField3DUtils::apply (UtilitiesDataTypes/HField3DUtils.txx:734-752)
__global__ void __launch_bounds__(kThreads)
    k_apply(const float *__restrict__ img, const float *__restrict__ hx, const float *__restrict__ hy,
            const float *__restrict__ hz, float *__restrict__ out, Dims d, float bg) {
  early_entry();
  Voxel vx;
  if (!voxel_of(d, vx)) return;
  const long i = vx.i;
  out[i] = trilerp_scalar(img, d, hx[i], hy[i], hz[i], bg);
}

// the spacing, its float divisors 2 sp (f2) and sp (f1) or their reciprocals,
// and how all six divide (the least of DivD::as)
struct AxisDiv {
  int as;
  float f2[3], f1[3];
  double s[3];
};
inline AxisDiv axis_div(const Spacing &sp) {
  AxisDiv a{2, {}, {}, {sp.x, sp.y, sp.z}};
  DivD c2[3], c1[3];
  for (int c = 0; c < 3; ++c) {
    c2[c] = make_div(2.0 * a.s[c]);
    c1[c] = make_div(a.s[c]);
    a.as = c2[c].as < a.as ? c2[c].as : a.as;
    a.as = c1[c].as < a.as ? c1[c].as : a.as;
  }
  for (int c = 0; c < 3; ++c) {  // a power of two is a float too
    a.f2[c] = a.as == 2 ? c2[c].fr : c2[c].fd;
    a.f1[c] = a.as == 2 ? c1[c].fr : c1[c].fd;
  }
  return a;
}

// Array3DUtils::computeGradient (Array3DUtils.txx:783-900). DOUBLE: spacings
// that are no floats. One kernel that chose per difference among the three
// kinds took 16.0 us at 128^3 with those and 49.7 at 160 x 180 x 200, this
// one 13.7 and 42.0; float spacings, all six values fetched before the
// arithmetic, 11.5 and 33.6 (10.8 and 38.0).
template <bool DOUBLE>
__global__ void __launch_bounds__(kThreads)
    k_gradient(const float *__restrict__ a, float *__restrict__ gx, float *__restrict__ gy,
               float *__restrict__ gz, Dims d, AxisDiv q, int wrap) {
  early_entry();
  Voxel vx;
  if (!voxel_of(d, vx)) return;
  const long i = vx.i;
  const int pos[3] = {vx.x, vx.y, vx.z};
  const int n[3] = {d.nx, d.ny, d.nz};
  const long stride[3] = {1, d.nx, (long)d.nx * d.ny};
  float *g[3] = {gx, gy, gz};
  if constexpr (DOUBLE) {
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      float r;
      if (pos[c] > 0 && pos[c] < n[c] - 1) {
        r = __double2float_rn((double)fsub(a[i + stride[c]], a[i - stride[c]]) / (2.0 * q.s[c]));
      } else if (wrap) {
        const long ip = pos[c] == n[c] - 1 ? i - (long)(n[c] - 1) * stride[c] : i + stride[c];
        const long im = pos[c] == 0 ? i + (long)(n[c] - 1) * stride[c] : i - stride[c];
        r = __double2float_rn((double)fsub(a[ip], a[im]) / (2.0 * q.s[c]));
      } else if (pos[c] == 0) {
        r = __double2float_rn((double)fsub(a[i + stride[c]], a[i]) / q.s[c]);
      } else {
        r = __double2float_rn((double)fsub(a[i], a[i - stride[c]]) / q.s[c]);
      }
      g[c][i] = r;
    }
    return;
  }
  float diff[3];
  bool central[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const bool lo = pos[c] == 0, hi = pos[c] == n[c] - 1;
    const long around = (long)(n[c] - 1) * stride[c];
    const long ip = hi ? (wrap ? i - around : i) : i + stride[c];
    const long im = lo ? (wrap ? i + around : i) : i - stride[c];
    central[c] = wrap || !(lo || hi);
    diff[c] = fsub(a[ip], a[im]);
  }
  if (q.as == 2) {
#pragma unroll
    for (int c = 0; c < 3; ++c) g[c][i] = fmul(diff[c], central[c] ? q.f2[c] : q.f1[c]);
  } else {
#pragma unroll
    for (int c = 0; c < 3; ++c) g[c][i] = fdiv(diff[c], central[c] ? q.f2[c] : q.f1[c]);
  }
}

// composeHV (dir=+1, HField3DUtils.txx:436-455) / composeHVInv (dir=-1,
// :461-480): h(x) = g(x +- (scale*v(x))/sp)
__global__ void __launch_bounds__(kThreads)
    k_compose_hv(const float *__restrict__ gx, const float *__restrict__ gy, const float *__restrict__ gz,
                 const float *__restrict__ vx, const float *__restrict__ vy, const float *__restrict__ vz,
                 float *__restrict__ ox, float *__restrict__ oy, float *__restrict__ oz, Dims d,
                 DivF q0, DivF q1, DivF q2, int dir, int bgs, const float *__restrict__ scale_ptr,
                 float scale_val) {
  early_entry();
  Voxel vox;
  if (!voxel_of(d, vox)) return;
  const long i = vox.i;
  const int x = vox.x, y = vox.y, z = vox.z;
  const float scale = scale_ptr ? *scale_ptr : scale_val;
  const float dx = fdivq(fmul(vx[i], scale), q0);
  const float dy = fdivq(fmul(vy[i], scale), q1);
  const float dz = fdivq(fmul(vz[i], scale), q2);
  float px, py, pz;
  if (dir > 0) {
    px = fadd(__int2float_rn(x), dx); py = fadd(__int2float_rn(y), dy); pz = fadd(__int2float_rn(z), dz);
  } else {
    px = fsub(__int2float_rn(x), dx); py = fsub(__int2float_rn(y), dy); pz = fsub(__int2float_rn(z), dz);
  }
  float rx, ry, rz;
  trilerp_vector(gx, gy, gz, d, px, py, pz, bgs, 1.0f, rx, ry, rz);
  ox[i] = rx;
  oy[i] = ry;
  oz[i] = rz;
}

// composeVH (dir=+1) / composeVHInv (dir=-1, HField3DUtils.txx:405-430):
// h(x) = g(x) +- (scale*v)(g(x))/sp
__global__ void __launch_bounds__(kThreads)
    k_compose_vh(const float *__restrict__ vx, const float *__restrict__ vy, const float *__restrict__ vz,
                 const float *__restrict__ gx, const float *__restrict__ gy, const float *__restrict__ gz,
                 float *__restrict__ ox, float *__restrict__ oy, float *__restrict__ oz, Dims d,
                 DivF q0, DivF q1, DivF q2, int dir, int bgs, const float *__restrict__ scale_ptr,
                 float scale_val) {
  early_entry();
  Voxel vox;
  if (!voxel_of(d, vox)) return;
  const long i = vox.i;
  const float scale = scale_ptr ? *scale_ptr : scale_val;
  const float g0 = gx[i], g1 = gy[i], g2 = gz[i];
  float hx, hy, hz;
  trilerp_vector(vx, vy, vz, d, g0, g1, g2, bgs, scale, hx, hy, hz);
  hx = fdivq(hx, q0); hy = fdivq(hy, q1); hz = fdivq(hz, q2);
  if (dir <= 0) {  // a / -s = -(a / s) exactly in round-to-nearest
    hx = -hx; hy = -hy; hz = -hz;
  }
  ox[i] = fadd(hx, g0);
  oy[i] = fadd(hy, g1);
  oz[i] = fadd(hz, g2);
}

}  // namespace

cudaError_t launch_apply(const float *img, const float *hx, const float *hy, const float *hz,
                         float *out, Dims d, float bg, cudaStream_t s) {
  launch_early(k_apply, row_grid(d), kThreads, 0, s, img, hx, hy, hz, out, d, bg);
  return cudaGetLastError();
}

cudaError_t launch_gradient(const float *a, float *gx, float *gy, float *gz, Dims d, Spacing sp,
                            int wrap, cudaStream_t s) {
  const AxisDiv q = axis_div(sp);
  if (q.as)
    launch_early(k_gradient<false>, row_grid(d), kThreads, 0, s, a, gx, gy, gz, d, q, wrap);
  else
    launch_early(k_gradient<true>, row_grid(d), kThreads, 0, s, a, gx, gy, gz, d, q, wrap);
  return cudaGetLastError();
}

cudaError_t launch_compose_hv(const float *const g[3], const float *const v[3], float *const o[3],
                              Dims d, Spacing sp, int dir, int bgs, const float *scale_ptr,
                              float scale_val, cudaStream_t s) {
  launch_early(k_compose_hv, row_grid(d), kThreads, 0, s, g[0], g[1], g[2], v[0], v[1], v[2], o[0],
               o[1], o[2], d, make_divf((float)sp.x), make_divf((float)sp.y),
               make_divf((float)sp.z), dir, bgs, scale_ptr, scale_val);
  return cudaGetLastError();
}

cudaError_t launch_compose_vh(const float *const v[3], const float *const g[3], float *const o[3],
                              Dims d, Spacing sp, int dir, int bgs, const float *scale_ptr,
                              float scale_val, cudaStream_t s) {
  launch_early(k_compose_vh, row_grid(d), kThreads, 0, s, v[0], v[1], v[2], g[0], g[1], g[2], o[0],
               o[1], o[2], d, make_divf((float)sp.x), make_divf((float)sp.y),
               make_divf((float)sp.z), dir, bgs, scale_ptr, scale_val);
  return cudaGetLastError();
}

}  // namespace aw
