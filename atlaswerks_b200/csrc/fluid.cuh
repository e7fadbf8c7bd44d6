// fluid.cuh — the fluid operator L = -alpha*Lap - beta*grad(div) + gamma and
// its inverse, applied in Fourier space by three fused kernels:
//
//   xy-forward  one CTA per (z-slab, component): producer (a field, or the
//               greedy/LDMM body force computed on the fly) -> real-to-complex
//               FFT along x (two real rows packed per complex line) -> FFT
//               along y -> half spectrum to HBM.
//   z-solve     one CTA per tile of (ky,kx) columns, all three components:
//               FFT along z -> per-wavenumber 3x3 solve (or multiply) with
//               1/N scaling -> inverse FFT along z -> back to HBM.
//   xy-inverse  one CTA per (z-slab, component): inverse FFT along y ->
//               complex-to-real along x -> consumer epilogue (store, or the
//               LDMM velocity update).
//
// The half spectrum (3 x nz x ny x (nx/2+1) complex64, or the slabs that
// fluid_any.cuh describes) makes two HBM round trips instead of the six of
// a pass-per-axis transform. fluid_fast.cu has the kernels for axes that
// are powers of two in [16, 256], fluid_any.cu those for any other grid.
#pragma once

#include <cuda.h>

#include "aw_common.cuh"
#include "fft_smem.cuh"
#include "fluid_any.cuh"

namespace aw {

struct FluidPlan {
  Dims d;
  Spacing sp;
  float alpha, beta, gamma;
  int nxh;
  FFTAxis ax, ay, az;        // register path: the axes' twiddle tables
  float2 *tw;                // device twiddle tables (x | y | z)
  float *lut;                // register path's LUT: cos x | sin x | cos y | sin y | cos z | sin z
  float2 *spec;              // device half spectrum
  // any-size path (fluid_any.cu): its plan (host) and its tables (device).
  // Slabs that do not fit one CTA's shared memory run an x and a y pass
  // through the spectrum in HBM (split), on pairs_per_batch row pairs and
  // cols_per_batch columns per CTA; the z pass takes zcols_per_cta columns.
  AnyPlan *any;
  uint32_t *any_tables;
  int split;
  int pairs_per_batch, cols_per_batch, zcols_per_cta;
  int device;
  // register-FFT path (fluid_fast.cu): power-of-two axes
  int fast;
  int fast_kq;               // (ky,kx) columns per z-pass CTA
  size_t fast_smem_xy, fast_smem_z;
  int *status;               // device status word: bounded waits that timed out
  int fast_tma;              // z-pass tiles moved by TMA tensor copies
  CUtensorMap spec_map;      // spectrum as [3][nz][2*ny*nxh] floats, 128B swizzle
};

// --- producers for the forward pass ----------------------------------------
// plain vector field input
// kPairs: row pairs whose loads the any-size path issues together
struct SrcField {
  static constexpr int kPairs = 4;
  const float *c[3];
  // slab z of component comp: the rows y and y + H at x, zero past the last row
  struct Slab {
    const float *f;
    int nx, ny, H;
    AW_D float2 pair(int x, int y) const {
      const int o = y * nx + x, y1 = y + H;
      const float a = __ldg(f + o), b = __ldg(f + (y1 < ny ? o + H * nx : o));
      return make_float2(a, y1 < ny ? b : 0.f);
    }
  };
  AW_D Slab at_slab(int comp, int z, int H, const Dims &d) const {
    return Slab{(comp == 0 ? c[0] : comp == 1 ? c[1] : c[2]) + d.idx(0, 0, z), d.nx, d.ny, H};
  }
  // rows y0 and y0+1 of slab z at x = t + TX*j, j < E, as (row y0, row y0+1)
  template <int E, int TX>
  AW_D void row_pair(int comp, int t, int y0, int z, const Dims &d, float2 *v) const {
    const float *r0 = (comp == 0 ? c[0] : comp == 1 ? c[1] : c[2]) + d.idx(t, y0, z);
    const float *r1 = r0 + d.nx;
#pragma unroll
    for (int j = 0; j < E; ++j) v[j] = make_float2(__ldg(r0 + TX * j), __ldg(r1 + TX * j));
  }
};

// body force f_c = d/dc(G) * M, with M = A - G (mode 1, greedy: G = I0(h),
// A = I1), M = A (mode 0, LDMM IterateNew: G = J0_{t-1}, A = splatted
// residual) or M = (G - A) * B (mode 2, LDMM IterateOrig: G = I0(h),
// A = JT_t, B = JacDet_t; LDMMIteratorCPU.cxx:447-452). The gradient is
// Array3DUtils::computeGradient with wrap = false (Array3DUtils.txx:783-900):
// central differences / (2 sp), one-sided at the borders, the float
// difference divided in double.
struct SrcForce {
  static constexpr int kPairs = 2;
  const float *G;
  const float *A;
  const float *B;
  int mode;
  DivD c2[3], c1[3];  // 2 sp and sp per axis
  // how all six divisors divide (DivD::as, the least of theirs), with the
  // float divisors (1) or reciprocals (2) at hand: one uniform choice and no
  // lookup of the whole divisor a voxel
  int as;
  float f2[3], f1[3];
  AW_D float grad(float diff, int comp, bool interior) const {
    if (as == 2) return fmul(diff, interior ? f2[comp] : f1[comp]);
    if (as == 1) return fdiv(diff, interior ? f2[comp] : f1[comp]);
    return __double2float_rn(ddiv((double)diff, interior ? c2[comp] : c1[comp]));
  }
  // M from preloaded values (b is read only in mode 2)
  AW_D float mismatch_v(float g0, float a, float b) const {
    return mode == 0 ? a : (mode == 1 ? -fsub(g0, a) : fmul(fsub(g0, a), b));
  }
  // One voxel. The neighbours are clamped to the voxel itself at the
  // borders (G[1] - G[0] at the first, G[n-1] - G[n-2] at the last; every
  // axis has n >= 2), so every load is issued before the arithmetic, with
  // no branch between them.
  AW_D float value(int comp, int x, int y, int z, const Dims &d) const {
    const long i = d.idx(x, y, z);
    int pos, n;
    long stride;
    if (comp == 0) { pos = x; n = d.nx; stride = 1; }
    else if (comp == 1) { pos = y; n = d.ny; stride = d.nx; }
    else { pos = z; n = d.nz; stride = (long)d.nx * d.ny; }
    const long ihi = pos < n - 1 ? i + stride : i, ilo = pos > 0 ? i - stride : i;
    const float g0 = __ldg(G + i), gh = __ldg(G + ihi), gl = __ldg(G + ilo), a = __ldg(A + i);
    const float b = mode == 2 ? __ldg(B + i) : 0.f;
    const float g = grad(fsub(gh, gl), comp, pos > 0 && pos < n - 1);
    return fmul(g, mismatch_v(g0, a, b));
  }
  // Slab z of component comp: the rows y and y + H at x, as value() forms
  // them, from offsets within the slab; zero past the last row. Every load
  // of the pair is issued before the arithmetic.
  struct Slab {
    const SrcForce *s;
    const float *g, *a, *b;  // the slab's first voxel
    int comp, nx, ny, H;
    int lo, hi;              // z: the neighbouring slabs' offsets
    bool in;                 // z: central difference
    AW_D float2 pair(int x, int y) const {
      const bool two = y + H < ny;
      const int y1 = two ? y + H : y, o0 = y * nx + x, o1 = y1 * nx + x;
      int l0 = lo, h0 = hi, l1 = lo, h1 = hi;
      bool in0 = in, in1 = in;
      if (comp == 0) {
        l0 = l1 = x > 0 ? -1 : 0;
        h0 = h1 = x < nx - 1 ? 1 : 0;
        in0 = in1 = x > 0 && x < nx - 1;
      } else if (comp == 1) {
        l0 = y > 0 ? -nx : 0;
        h0 = y < ny - 1 ? nx : 0;
        in0 = y > 0 && y < ny - 1;
        l1 = y1 > 0 ? -nx : 0;
        h1 = y1 < ny - 1 ? nx : 0;
        in1 = y1 > 0 && y1 < ny - 1;
      }
      const float g0 = __ldg(g + o0), gh0 = __ldg(g + o0 + h0), gl0 = __ldg(g + o0 + l0);
      const float g1 = __ldg(g + o1), gh1 = __ldg(g + o1 + h1), gl1 = __ldg(g + o1 + l1);
      const float a0 = __ldg(a + o0), a1 = __ldg(a + o1);
      float b0 = 0.f, b1 = 0.f;
      if (s->mode == 2) {
        b0 = __ldg(b + o0);
        b1 = __ldg(b + o1);
      }
      const float v0 = fmul(s->grad(fsub(gh0, gl0), comp, in0), s->mismatch_v(g0, a0, b0));
      const float v1 = fmul(s->grad(fsub(gh1, gl1), comp, in1), s->mismatch_v(g1, a1, b1));
      return make_float2(v0, two ? v1 : 0.f);
    }
  };
  AW_D Slab at_slab(int comp, int z, int H, const Dims &d) const {
    const long o = d.idx(0, 0, z);
    const int sl = d.nx * d.ny;
    return Slab{this, G + o,  A + o, B + o, comp, d.nx, d.ny, H, z > 0 ? -sl : 0, z < d.nz - 1 ? sl : 0,
                z > 0 && z < d.nz - 1};
  }
  // Rows y0 and y0+1 of slab z at x = t + TX*j, j < E, as (row y0, row
  // y0+1): the same values as value(), from row pointers formed once and one
  // code path per component. Every load of the row pair (G and its
  // neighbours, A, and B in mode 2; of each chunk of it in 256-wide rows) is
  // issued before any arithmetic that depends on one, so the pair costs one
  // round trip to L2, not one per array. Needs nx, ny, nz >= 3, an even ny, TX * E = nx and the TX lanes
  // of a line consecutive within a warp, every lane of the warp calling it
  // (the x neighbours come by shuffles).
  template <int E, int TX>
  AW_D void row_pair(int comp, int t, int y0, int z, const Dims &d, float2 *v) const {
    // the values of each array per lane in flight at once: the whole row
    // pair up to E = 4, chunks of two above (a 256-wide row would spill)
    constexpr int C = E <= 4 ? E : 2;
    const long i0 = d.idx(t, y0, z);
    const int nx = d.nx;
    const float *g0p = G + i0, *g1p = g0p + nx, *a0p = A + i0, *b0p = B + i0;
    float a0[C], a1[C], b0[C], b1[C];
    // A (and B) of chunk j0 .. j0 + C - 1
    auto load_ab = [&](int j0) {
#pragma unroll
      for (int c = 0; c < C; ++c) {
        const int o = TX * (j0 + c);
        a0[c] = __ldg(a0p + o);
        a1[c] = __ldg(a0p + o + nx);
      }
      if (mode == 2) {
#pragma unroll
        for (int c = 0; c < C; ++c) {
          const int o = TX * (j0 + c);
          b0[c] = __ldg(b0p + o);
          b1[c] = __ldg(b0p + o + nx);
        }
      } else {
#pragma unroll
        for (int c = 0; c < C; ++c) b0[c] = b1[c] = 0.f;
      }
    };
    if (comp == 0) {
      // the line covers the row (TX * E = nx): x +- 1 is held by the
      // neighbouring lane at the same j, or by the line's first / last lane
      // at j +- 1, so the neighbours come by shuffles instead of loads
      float r0[E], r1[E];
#pragma unroll
      for (int j = 0; j < E; ++j) {
        r0[j] = __ldg(g0p + TX * j);
        r1[j] = __ldg(g1p + TX * j);
      }
      const unsigned full = 0xffffffffu;
      const int up = (t + 1) & (TX - 1), dn = (t - 1) & (TX - 1);
#pragma unroll
      for (int j0 = 0; j0 < E; j0 += C) {
        load_ab(j0);
#pragma unroll
        for (int c = 0; c < C; ++c) {
          const int j = j0 + c;
          const int jn = j + 1 < E ? j + 1 : j, jp = j > 0 ? j - 1 : j;
          const float n0 = __shfl_sync(full, r0[j], up, TX), n1 = __shfl_sync(full, r1[j], up, TX);
          const float w0 = __shfl_sync(full, r0[jn], 0, TX), w1 = __shfl_sync(full, r1[jn], 0, TX);
          const float p0 = __shfl_sync(full, r0[j], dn, TX), p1 = __shfl_sync(full, r1[j], dn, TX);
          const float q0 = __shfl_sync(full, r0[jp], TX - 1, TX),
                      q1 = __shfl_sync(full, r1[jp], TX - 1, TX);
          const int x = t + TX * j;
          const bool first = x == 0, last = x == nx - 1, in = !first && !last;
          // G[x + hi] and G[x + lo], hi = 0 at the last voxel, lo = 0 at the first
          const float h0 = last ? r0[j] : (t == TX - 1 ? w0 : n0);
          const float h1 = last ? r1[j] : (t == TX - 1 ? w1 : n1);
          const float l0 = first ? r0[j] : (t == 0 ? q0 : p0);
          const float l1 = first ? r1[j] : (t == 0 ? q1 : p1);
          v[j] = make_float2(fmul(grad(fsub(h0, l0), 0, in), mismatch_v(r0[j], a0[c], b0[c])),
                             fmul(grad(fsub(h1, l1), 0, in), mismatch_v(r1[j], a1[c], b1[c])));
        }
      }
    } else if (comp == 1) {
      // y0 - 1 (or y0 at the first row) and y0 + 2 (or y0 + 1 at the last)
      const int lo = y0 > 0 ? -nx : 0, hi = y0 + 2 < d.ny ? 2 * nx : nx;
      const bool in0 = y0 > 0, in1 = y0 + 2 < d.ny;
#pragma unroll
      for (int j0 = 0; j0 < E; j0 += C) {
        float g0[C], g1[C], gl[C], gh[C];
#pragma unroll
        for (int c = 0; c < C; ++c) {
          const int o = TX * (j0 + c);
          g0[c] = __ldg(g0p + o);
          g1[c] = __ldg(g1p + o);
          gl[c] = __ldg(g0p + o + lo);
          gh[c] = __ldg(g0p + o + hi);
        }
        load_ab(j0);
#pragma unroll
        for (int c = 0; c < C; ++c) {
          // row y0: G[y0+1] - G[y0-1], or G[1] - G[0] (lo = 0);
          // row y0+1: G[y0+2] - G[y0], or G[ny-1] - G[ny-2] (hi = nx)
          const float d0 = fsub(g1[c], gl[c]);
          const float d1 = fsub(gh[c], g0[c]);
          v[j0 + c] = make_float2(fmul(grad(d0, 1, in0), mismatch_v(g0[c], a0[c], b0[c])),
                                  fmul(grad(d1, 1, in1), mismatch_v(g1[c], a1[c], b1[c])));
        }
      }
    } else {
      const long sl = (long)nx * d.ny;
      const long lo = z > 0 ? -sl : 0, hi = z < d.nz - 1 ? sl : 0;
      const bool in = z > 0 && z < d.nz - 1;
#pragma unroll
      for (int j0 = 0; j0 < E; j0 += C) {
        float g0[C], g1[C], h0[C], l0[C], h1[C], l1[C];
#pragma unroll
        for (int c = 0; c < C; ++c) {
          const int o = TX * (j0 + c);
          g0[c] = __ldg(g0p + o);
          g1[c] = __ldg(g1p + o);
          h0[c] = __ldg(g0p + o + hi);
          l0[c] = __ldg(g0p + o + lo);
          h1[c] = __ldg(g1p + o + hi);
          l1[c] = __ldg(g1p + o + lo);
        }
        load_ab(j0);
#pragma unroll
        for (int c = 0; c < C; ++c) {
          const float d0 = fsub(h0[c], l0[c]);
          const float d1 = fsub(h1[c], l1[c]);
          v[j0 + c] = make_float2(fmul(grad(d0, 2, in), mismatch_v(g0[c], a0[c], b0[c])),
                                  fmul(grad(d1, 2, in), mismatch_v(g1[c], a1[c], b1[c])));
        }
      }
    }
  }
};
inline SrcForce make_force(const float *G, const float *A, int mode, const Spacing &sp,
                           const float *B = nullptr) {
  SrcForce f;
  f.G = G;
  f.A = A;
  f.B = B;
  f.mode = mode;
  const double s[3] = {sp.x, sp.y, sp.z};
  f.as = 2;
  for (int c = 0; c < 3; ++c) {
    f.c2[c] = make_div(2.0 * s[c]);
    f.c1[c] = make_div(s[c]);
    for (const DivD *q : {&f.c2[c], &f.c1[c]}) f.as = q->as < f.as ? q->as : f.as;
  }
  for (int c = 0; c < 3; ++c) {
    // a power of two is a float too, so the least kind serves all six
    f.f2[c] = f.as == 2 ? f.c2[c].fr : f.c2[c].fd;
    f.f1[c] = f.as == 2 ? f.c1[c].fr : f.c1[c].fd;
  }
  return f;
}

// --- consumers for the inverse pass ----------------------------------------
// A kernel stores component `comp` through dst.bind(comp): the component's
// pointer picked once (no indexed parameter array) and any per-launch
// factors formed once.
struct DstFieldBound {
  float *c;
  AW_D void store(long i, float v) const { c[i] = v; }
};
struct DstField {
  static constexpr bool kReads = false;
  float *c[3];
  AW_D DstFieldBound bind(int comp) const {
    return DstFieldBound{comp == 0 ? c[0] : comp == 1 ? c[1] : c[2]};
  }
};

// -K f: the shooting velocities (LDMMAdShootingIteratorCPU.cxx:256-261,
// 291-296 scale K f by -1, an exact sign flip)
struct DstNegBound {
  float *c;
  AW_D void store(long i, float v) const { c[i] = -v; }
};
struct DstNeg {
  static constexpr bool kReads = false;
  float *c[3];
  AW_D DstNegBound bind(int comp) const {
    return DstNegBound{comp == 0 ? c[0] : comp == 1 ? c[1] : c[2]};
  }
};

// LDMM velocity update v = vfac * v + ufac * u (LDMMIteratorCPU::updateVelocity,
// LDMM/LDMMIteratorCPU.cxx:177-190) with vfac = 1 - 2*eps and
// ufac = 2*eps / sigma^2 formed from the device-resident step eps, float
// arithmetic in the reference's order (LDMMIteratorCPU.cxx:606-609).
struct DstAxpbyBound {
  float *c;
  float vfac, ufac;
  AW_D void store(long i, float u) const { c[i] = fadd(fmul(vfac, c[i]), fmul(ufac, u)); }
  // n elements: every old value is read before any is written
  template <int N>
  AW_D void store_n(const long (&i)[N], const float (&u)[N]) const {
    float old[N];
#pragma unroll
    for (int j = 0; j < N; ++j) old[j] = c[i[j]];
#pragma unroll
    for (int j = 0; j < N; ++j) c[i[j]] = fadd(fmul(vfac, old[j]), fmul(ufac, u[j]));
  }
  // the same, without the elements whose index is negative
  template <int N>
  AW_D void store_some(const long (&i)[N], const float (&u)[N]) const {
    float old[N];
#pragma unroll
    for (int j = 0; j < N; ++j) old[j] = i[j] >= 0 ? c[i[j]] : 0.f;
#pragma unroll
    for (int j = 0; j < N; ++j)
      if (i[j] >= 0) c[i[j]] = fadd(fmul(vfac, old[j]), fmul(ufac, u[j]));
  }
};
struct DstAxpby {
  static constexpr bool kReads = true;
  float *c[3];
  const float *step;
  float sigma;
  // the step read once per thread, the two factors formed once
  AW_D DstAxpbyBound bind(int comp) const {
    const float eps = *step;
    const float vfac = fsub(1.0f, fmul(2.0f, eps));
    const float ufac = fdiv(fmul(2.0f, eps), fmul(sigma, sigma));
    return DstAxpbyBound{comp == 0 ? c[0] : comp == 1 ? c[1] : c[2], vfac, ufac};
  }
};

// The greedy update h'(x) = h(x + eps v(x)/sp) the inverse pass can apply
// itself (fluid_inverse_compose): h in, h' out, the device-resident step,
// the spacing divisors.
struct ComposeArgs {
  const float *hx, *hy, *hz;
  float *ox, *oy, *oz;
  const float *step;
  DivF q0, q1, q2;
  int fast;  // 1: float-tree interpolation (trilerp_vector<true>)
};

// host API (fluid.cu)
int fluid_plan_create(FluidPlan *p, int nx, int ny, int nz, double spx, double spy, double spz,
                      float alpha, float beta, float gamma);
void fluid_plan_destroy(FluidPlan *p);

cudaError_t fluid_forward_field(const FluidPlan &p, const float *fx, const float *fy,
                                const float *fz, cudaStream_t s);
cudaError_t fluid_forward_force(const FluidPlan &p, const float *G, const float *A, int diff,
                                cudaStream_t s);
// force (G - A) * B * grad G (mode 2)
cudaError_t fluid_forward_force_jac(const FluidPlan &p, const float *G, const float *A,
                                    const float *B, cudaStream_t s);
cudaError_t fluid_solve(const FluidPlan &p, int inverse, cudaStream_t s);
// shapes of the shared-memory (any-size) path; fluid_get_shapes returns 0 on
// the register path, whose shapes are fixed
int fluid_get_shapes(const FluidPlan &p, int *P, int *Q, int *K);
cudaError_t fluid_set_shapes(FluidPlan *p, int P, int Q, int K);
cudaError_t fluid_autotune(FluidPlan *p, cudaStream_t s);
// the plan's status word: *timed_out = 1 when a transform kernel's bounded
// wait ran out since the last call; the word is cleared (stream-ordered)
cudaError_t fluid_take_status(FluidPlan *p, int *timed_out, cudaStream_t s);
// one CTA whose bounded wait (polls polls) on an mbarrier that nothing
// arrives on runs out and records the timeout in the plan's status word
cudaError_t fluid_wait_selftest(const FluidPlan &p, int polls, cudaStream_t s);
cudaError_t fluid_inverse_store(const FluidPlan &p, float *ox, float *oy, float *oz,
                                cudaStream_t s);
cudaError_t fluid_inverse_store_neg(const FluidPlan &p, float *ox, float *oy, float *oz,
                                    cudaStream_t s);
// v = K f never leaves the chip: h' = h(x + eps v/sp) from the inverse pass
// itself (power-of-two grids: the register-FFT path); cudaErrorNotSupported
// on other grids, where the caller stores v and updates separately
cudaError_t fluid_inverse_compose(const FluidPlan &p, const ComposeArgs &a, cudaStream_t s);
cudaError_t fluid_inverse_axpby(const FluidPlan &p, float *vx, float *vy, float *vz,
                                const float *step, float sigma, cudaStream_t s);

}  // namespace aw
