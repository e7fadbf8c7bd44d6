// fluid.cu — fused FFT kernels of the fluid operator solve (see fluid.cuh).
//
// Reference behaviour (Algorithms/Common/DiffOper.cxx:825-905 on the CPU,
// CUDACommon/src/cudaFFTSolver.cu:675-704 on the old GPU path): the force is
// scaled by 1/N, transformed, multiplied per wavenumber by L(k)^-1 (or L(k)),
// and transformed back, with
//   lambda = -alpha*(cx+cy+cz) + gamma,  L_ii = lambda - beta*c_i,
//   L_ij = beta*s_i*s_j,  c = (2cos(2 pi k/n) - 2)/sp^2,  s = sin(2 pi k/n)/sp
// (LUT: DiffOper.cxx:590-639; Cholesky: DiffOper.cxx:1005-1083). Here the
// 1/N scaling is folded into the per-wavenumber step.
#include <cudaTypedefs.h>

#include <cmath>
#include <cstring>
#include <map>
#include <mutex>
#include <new>
#include <tuple>
#include <vector>

#include "bulk.cuh"
#include "fluid.cuh"
#include "tma_host.cuh"
#include "fluid_fast.cuh"

namespace aw {

namespace {

void fill_twiddles(int n, std::vector<float2> &out) {
  for (int m = 0; m < n; ++m) {
    const double a = -2.0 * M_PI * (double)m / (double)n;
    out.push_back(make_float2((float)std::cos(a), (float)std::sin(a)));
  }
}

// reference LUT, computed in double and stored as float like DiffOperT<float>
void fill_lut(int n, double sp, std::vector<float> &out) {
  const double s = 2.0 * M_PI / n;
  for (int k = 0; k < n; ++k) out.push_back((float)((2.0 * std::cos(s * k) - 2.0) / (sp * sp)));
  for (int k = 0; k < n; ++k) out.push_back((float)(std::sin(s * k) / sp));
}

// TMA descriptor of the spectrum for the z-pass: a 3D float tensor
// {2*ny*nxh, nz, 3} read and written in boxes {2*Kq, nz, 1} = one row per
// kz of 16 columns (128 bytes, 128-byte swizzle) or 8 (64 bytes, 64-byte
// swizzle) in shared memory
bool encode_spec_map(FluidPlan *p) {
  const PFN_cuTensorMapEncodeTiled encode = tensor_map_encoder();
  if (!encode) return false;
  const cuuint64_t ncols = (cuuint64_t)p->d.ny * p->nxh;
  const cuuint64_t dims[3] = {2 * ncols, (cuuint64_t)p->d.nz, 3};
  const cuuint64_t strides[2] = {2 * ncols * sizeof(float), 2 * ncols * sizeof(float) * p->d.nz};
  const cuuint32_t box[3] = {(cuuint32_t)(2 * p->fast_kq), (cuuint32_t)p->d.nz, 1};
  const cuuint32_t estr[3] = {1, 1, 1};
  const size_t row = box[0] * sizeof(float);
  if ((row != 128 && row != 64) || box[1] > 256 || strides[0] % 16) return false;
  return encode(&p->spec_map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, p->spec, dims, strides, box, estr,
                CU_TENSOR_MAP_INTERLEAVE_NONE,
                row == 128 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B,
                CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// The register path's z-pass tile width (16 or 8 columns) by timing: after
// one untimed launch, three alternating L^-1 / L launches (the spectrum
// keeps its scale) of each on a zeroed spectrum; the faster is kept per
// (grid, device) for the process. The arithmetic of a column does not
// depend on the width.
std::mutex g_zq_mu;
std::map<std::tuple<int, int, int, int>, int> g_zq;

void tune_z_cols(FluidPlan *p) {
  const auto key = std::make_tuple(p->d.nx, p->d.ny, p->d.nz, p->device);
  {
    std::lock_guard<std::mutex> lock(g_zq_mu);
    auto it = g_zq.find(key);
    if (it != g_zq.end()) {
      p->fast_kq = it->second;
      p->fast_tma = encode_spec_map(p);
      return;
    }
  }
  const size_t bytes = sizeof(float2) * 3 * (size_t)p->d.nz * p->d.ny * p->nxh;
  if (cudaMemset(p->spec, 0, bytes) != cudaSuccess) return;
  cudaEvent_t e0, e1;
  if (cudaEventCreate(&e0) != cudaSuccess) return;
  if (cudaEventCreate(&e1) != cudaSuccess) {
    cudaEventDestroy(e0);
    return;
  }
  float best = 1e30f;
  int pick = 16;
  for (int q : {16, 8}) {
    p->fast_kq = q;
    p->fast_tma = encode_spec_map(p);
    fast_z_solve(*p, 1, 0);
    cudaEventRecord(e0, 0);
    for (int r = 0; r < 3; ++r) fast_z_solve(*p, r & 1, 0);
    cudaEventRecord(e1, 0);
    float ms = 0.f;
    if (cudaEventSynchronize(e1) != cudaSuccess || cudaEventElapsedTime(&ms, e0, e1) != cudaSuccess)
      break;
    if (ms < best) {
      best = ms;
      pick = q;
    }
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  p->fast_kq = pick;
  p->fast_tma = encode_spec_map(p);
  if (cudaGetLastError() != cudaSuccess) return;
  std::lock_guard<std::mutex> lock(g_zq_mu);
  g_zq[key] = pick;
}

// The shared-memory limit is an attribute of the kernel, shared by every
// plan on the device: only ever raise it, so a plan created later with a
// smaller footprint cannot invalidate the launches of a larger one.
std::mutex g_smem_mu;
std::map<std::pair<const void *, int>, size_t> g_smem;

cudaError_t set_smem(const void *kernel, size_t bytes) {
  int dev = 0;
  cudaGetDevice(&dev);
  std::lock_guard<std::mutex> lock(g_smem_mu);
  size_t &cur = g_smem[{kernel, dev}];
  if (bytes <= cur) return cudaSuccess;
  const cudaError_t e =
      cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  if (e == cudaSuccess) cur = bytes;
  return e;
}

// what a block's dynamic shared memory may take: the kernels' barrier lies
// before it, on 128 bytes with the alignment
size_t any_smem_limit(int device) {
  int maxsm = 0;
  cudaDeviceGetAttribute(&maxsm, cudaDevAttrMaxSharedMemoryPerBlockOptin, device);
  return (size_t)std::max(0, maxsm - 128);
}

// Launch shapes of the any-size path, into a. P row pairs and Q columns per
// CTA (split grids; a slab that fits one CTA is its own batch), K columns per
// z-pass CTA, taken up to a power of two between 8 and 32.
// Threads: the xy kernels' registers allow 768 threads on an SM, the z
// kernel's 1024: these are shared out over the CTAs that an SM gets, by
// its shared memory and by the grid.
// False: a kernel's shared memory would exceed maxsm. A slab in one CTA and a
// z tile of 16 columns of 512 always fit (fluid_plan_create splits the
// others); 32 columns do up to nz = 293.
bool any_shapes(const FluidPlan &p, AnyPlan *a, int P, int Q, int K, size_t maxsm) {
  int sms = 148;
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, p.device);
  auto threads = [&](size_t smem, long ctas, int budget, int lo, int hi) {
    const long by_smem = std::max<long>(1, (long)((227u * 1024u) / (smem + 1024)));
    const long per_sm = std::max<long>(1, std::min<long>(by_smem, (ctas + sms - 1) / sms));
    return (int)std::max<long>(lo, std::min<long>(hi, budget / per_sm / 32 * 32));
  };
  int q = 8;
  while (q < K && q < 32) q *= 2;
  any_set_z(a, q);
  a->threads_z = threads(a->smem_z, (a->z.pcols + q - 1) / q, 1024, 64, 256);
  a->smem_xy = any_smem_xy(a->xy);
  a->threads_xy = threads(a->smem_xy, 3L * p.d.nz, 768, 128, 768);
  any_set_split(a, P, Q, maxsm);
  const bool xy = p.split ? a->smem_x <= maxsm && any_smem_y(a->xy, Q) <= maxsm : a->smem_xy <= maxsm;
  return xy && a->smem_z <= maxsm;
}

cudaError_t any_configure(const AnyPlan &a, bool split) {
  for (const auto &k : any_kernels(a, split)) {
    const cudaError_t e = set_smem(k.first, k.second);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

// the any-size path's tables in one allocation, and the plan's device pointers
bool upload_any(FluidPlan *p, const AnyTables &t) {
  AnyPlan &a = *p->any;
  std::vector<uint32_t> all;  // the float4 tables first: 16-byte aligned
  auto words = [&](const void *v, size_t bytes) {
    const size_t at = all.size();
    all.resize(at + bytes / sizeof(uint32_t));
    std::memcpy(all.data() + at, v, bytes);
    return at;
  };
  const size_t lx = words(t.lutx.data(), t.lutx.size() * sizeof(float4));
  const size_t ly = words(t.luty.data(), t.luty.size() * sizeof(float4));
  const size_t lz = words(t.lutz.data(), t.lutz.size() * sizeof(float4));
  const size_t kxy = words(t.kxy.data(), t.kxy.size() * sizeof(uint32_t));
  const size_t cols = words(t.cols.data(), t.cols.size() * sizeof(uint32_t));
  const size_t packed = words(t.packed.data(), t.packed.size() * sizeof(uint32_t));
  if (cudaMalloc(&p->any_tables, all.size() * sizeof(uint32_t)) != cudaSuccess) return false;
  if (cudaMemcpy(p->any_tables, all.data(), all.size() * sizeof(uint32_t), cudaMemcpyHostToDevice) !=
      cudaSuccess)
    return false;
  const uint32_t *d = p->any_tables;
  a.z.lutx = reinterpret_cast<const float4 *>(d + lx);
  a.z.luty = reinterpret_cast<const float4 *>(d + ly);
  a.z.lutz = reinterpret_cast<const float4 *>(d + lz);
  a.z.kxy = d + kxy;
  a.xy.cols = d + cols;
  a.xy.packed = d + packed;
  a.xy.x.tw = p->ax.tw;
  a.xy.y.tw = p->ay.tw;
  a.z.z.tw = p->az.tw;
  a.xy.spec = a.z.spec = p->spec;
  a.xy.status = p->status;
  return true;
}

// autotuned shapes per (grid, device), kept for the life of the process
std::mutex g_tune_mu;
std::map<std::tuple<int, int, int, int>, std::tuple<int, int, int>> g_tuned;

}  // namespace

int fluid_get_shapes(const FluidPlan &p, int *P, int *Q, int *K) {
  *P = p.fast ? 0 : p.pairs_per_batch;
  *Q = p.fast ? 0 : p.cols_per_batch;
  *K = p.fast ? p.fast_kq : p.zcols_per_cta;
  return p.fast ? 0 : 1;
}

cudaError_t fluid_set_shapes(FluidPlan *p, int P, int Q, int K) {
  const int npairs = (p->d.ny + 1) / 2;
  if (p->fast) {
    // the register path: only the z-pass tile width, 16 or 8 columns
    if (P != 0 || Q != 0 || (K != 16 && K != 8)) return cudaErrorInvalidValue;
    p->fast_kq = K;
    p->fast_tma = encode_spec_map(p);
    return cudaSuccess;
  }
  if (P < 1 || P > npairs || Q < 1 || Q > p->nxh || K < 1 || K > 64) return cudaErrorInvalidValue;
  AnyPlan a = *p->any;  // a rejected shape leaves the plan as it is
  if (!any_shapes(*p, &a, P, Q, K, any_smem_limit(p->device))) return cudaErrorInvalidValue;
  const cudaError_t e = any_configure(a, p->split);
  if (e != cudaSuccess) return e;
  *p->any = a;
  p->pairs_per_batch = P;
  p->cols_per_batch = Q;
  p->zcols_per_cta = K;
  return cudaSuccess;
}

// The any-size path's autotuner: on split grids every combination of half,
// the heuristic and twice the heuristic row pairs and columns per CTA is
// timed on the forward + inverse xy pass, then 8, 16 and 32 columns per z
// CTA on the z pass (alternating L^-1 and L so the spectrum keeps its
// scale), each the mean of three launches after one untimed, on a zero field
// (the arithmetic is the same for every shape; only the distribution of
// lines over CTAs changes). The choice is kept per grid and device.
cudaError_t fluid_autotune(FluidPlan *p, cudaStream_t s) {
  if (p->fast) return cudaSuccess;
  const auto key = std::make_tuple(p->d.nx, p->d.ny, p->d.nz, p->device);
  {
    std::lock_guard<std::mutex> lock(g_tune_mu);
    auto it = g_tuned.find(key);
    if (it != g_tuned.end())
      return fluid_set_shapes(p, std::get<0>(it->second), std::get<1>(it->second),
                              std::get<2>(it->second));
  }
  const long n = p->d.n();
  float *f = nullptr;
  cudaError_t e = cudaMalloc(&f, sizeof(float) * 3 * n);
  if (e != cudaSuccess) {  // no room for the tuning field: keep the heuristic shapes
    cudaGetLastError();
    return cudaSuccess;
  }
  cudaEvent_t e0 = nullptr, e1 = nullptr;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  auto timed = [&](auto &&fn, float *ms) -> cudaError_t {
    cudaError_t r = fn();
    if (r != cudaSuccess) return r;
    cudaEventRecord(e0, s);
    for (int i = 0; i < 3 && r == cudaSuccess; ++i) r = fn();
    cudaEventRecord(e1, s);
    if (r == cudaSuccess) r = cudaEventSynchronize(e1);
    if (r == cudaSuccess) r = cudaEventElapsedTime(ms, e0, e1);
    return r;
  };
  float *c[3] = {f, f + n, f + 2 * n};
  // the shapes that the plan holds stand unless a candidate beats them
  const int P0 = p->pairs_per_batch, Q0 = p->cols_per_batch, K0 = p->zcols_per_cta;
  int bestP = P0, bestQ = Q0, bestK = K0;
  float best = 1e30f;
  if ((e = cudaMemsetAsync(f, 0, sizeof(float) * 3 * n, s)) == cudaSuccess) {
    for (int P : {P0 / 2, P0, 2 * P0})
      for (int Q : {Q0 / 2, Q0, 2 * Q0}) {
        if (!p->split) break;  // the whole slab is one batch
        if (fluid_set_shapes(p, P, Q, K0) != cudaSuccess) continue;
        float ms = 0.f;
        if ((e = timed([&]() {
               cudaError_t r = fluid_forward_field(*p, c[0], c[1], c[2], s);
               return r == cudaSuccess ? fluid_inverse_store(*p, c[0], c[1], c[2], s) : r;
             }, &ms)) != cudaSuccess)
          break;
        if (ms < best) {
          best = ms;
          bestP = P;
          bestQ = Q;
        }
      }
  }
  if (e == cudaSuccess) {
    best = 1e30f;
    int flip = 0;
    for (int K : {8, 16, 32}) {
      if (fluid_set_shapes(p, bestP, bestQ, K) != cudaSuccess) continue;
      float ms = 0.f;
      if ((e = timed([&]() { return fluid_solve(*p, (flip++ & 1) ? 0 : 1, s); }, &ms)) !=
          cudaSuccess)
        break;
      if (ms < best) {
        best = ms;
        bestK = K;
      }
    }
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cudaFree(f);
  if (e != cudaSuccess) return e;
  {
    std::lock_guard<std::mutex> lock(g_tune_mu);
    g_tuned[key] = std::make_tuple(bestP, bestQ, bestK);
  }
  return fluid_set_shapes(p, bestP, bestQ, bestK);
}

int fluid_plan_create(FluidPlan *p, int nx, int ny, int nz, double spx, double spy, double spz,
                      float alpha, float beta, float gamma) {
  std::memset(p, 0, sizeof(*p));
  if (nx < 2 || ny < 2 || nz < 2 || nx > 512 || ny > 512 || nz > 512) return 1;
  p->d = Dims{nx, ny, nz};
  p->sp = Spacing{spx, spy, spz};
  p->alpha = alpha;
  p->beta = beta;
  p->gamma = gamma;
  p->nxh = nx / 2 + 1;
  int dev = 0, maxsm = 0;
  cudaGetDevice(&dev);
  p->device = dev;
  cudaDeviceGetAttribute(&maxsm, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  if (fast_supported(nx) && fast_supported(ny) && fast_supported(nz)) {
    p->fast_kq = fast_z_cols();
    p->fast_smem_xy = fast_xy_smem(nx, ny);
    p->fast_smem_z = fast_z_smem(nz, 16);
    p->fast = p->fast_smem_xy <= (size_t)maxsm && p->fast_smem_z <= (size_t)maxsm;
  }
  AnyTables tab;
  if (!p->fast) {
    p->any = new (std::nothrow) AnyPlan();
    if (!p->any) return 3;
    if (!any_plan(p->any, &tab, p->d, p->sp, alpha, beta, gamma, false)) return 1;
    // a slab whose half spectrum does not fit one CTA: the split x / y passes
    const size_t limit = any_smem_limit(dev);
    if (any_smem_xy(p->any->xy) > limit) {
      p->split = 1;
      if (!any_plan(p->any, &tab, p->d, p->sp, alpha, beta, gamma, true)) return 1;
    }
    const int npairs = (ny + 1) / 2;
    p->pairs_per_batch = std::max(1, std::min(npairs, (2048 + nx - 1) / nx));
    p->cols_per_batch = std::max(1, std::min(p->nxh, p->split ? 32 : (2048 + ny - 1) / ny));
    p->zcols_per_cta = std::max(1, std::min(16, 3072 / (3 * nz)));
    if (!any_shapes(*p, p->any, p->pairs_per_batch, p->cols_per_batch, p->zcols_per_cta, limit))
      return 2;
  }
  const size_t spec_elems = p->fast ? 3 * (size_t)nz * ny * p->nxh
                                    : 3 * (size_t)nz * (size_t)p->any->xy.pcols;

  std::vector<float2> tw;
  fill_twiddles(nx, tw);
  fill_twiddles(ny, tw);
  fill_twiddles(nz, tw);
  std::vector<float> lut;
  if (p->fast) {
    fill_lut(nx, spx, lut);
    fill_lut(ny, spy, lut);
    fill_lut(nz, spz, lut);
  }
  if (cudaMalloc(&p->tw, tw.size() * sizeof(float2)) != cudaSuccess) return 3;
  if (p->fast && cudaMalloc(&p->lut, lut.size() * sizeof(float)) != cudaSuccess) return 3;
  if (cudaMalloc(&p->spec, sizeof(float2) * spec_elems) != cudaSuccess) return 3;
  if (cudaMalloc(&p->status, sizeof(int)) != cudaSuccess) return 3;
  cudaMemset(p->status, 0, sizeof(int));
  cudaMemcpy(p->tw, tw.data(), tw.size() * sizeof(float2), cudaMemcpyHostToDevice);
  if (p->fast) cudaMemcpy(p->lut, lut.data(), lut.size() * sizeof(float), cudaMemcpyHostToDevice);
  p->ax.tw = p->tw;
  p->ay.tw = p->tw + nx;
  p->az.tw = p->tw + nx + ny;
  if (p->any) {
    if (!upload_any(p, tab)) return 3;
    if (any_configure(*p->any, p->split) != cudaSuccess) return 4;
  }
  if (p->fast) p->fast_tma = encode_spec_map(p);
  if (p->fast && fast_configure(*p) != cudaSuccess) return 4;
  if (p->fast) tune_z_cols(p);
  if (!p->fast && fluid_autotune(p, 0) != cudaSuccess) return 4;
  return cudaGetLastError() == cudaSuccess ? 0 : 4;
}

namespace {

// The timeout path of the transform kernels, run on purpose: nothing ever
// arrives on this barrier, so every thread's bounded wait gives up after
// `polls` polls, the status word records it, and the CTA leaves together
// as a transform CTA does when its slab never lands. Nothing is in flight
// on the barrier when the CTA exits.
__global__ void k_wait_selftest(int *status, int polls) {
  __shared__ __align__(8) uint64_t mbar;
  if (threadIdx.x == 0) mbar_init(&mbar, 1);
  __syncthreads();
  const bool ok = mbar_wait(&mbar, 0, status, polls);
  (void)__syncthreads_or(!ok);
}

}  // namespace

cudaError_t fluid_wait_selftest(const FluidPlan &p, int polls, cudaStream_t s) {
  k_wait_selftest<<<1, 32, 0, s>>>(p.status, polls);
  return cudaGetLastError();
}

cudaError_t fluid_take_status(FluidPlan *p, int *timed_out, cudaStream_t s) {
  int v = 0;
  cudaError_t e = cudaMemcpyAsync(&v, p->status, sizeof(int), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return e;
  *timed_out = v == kStatusWaitTimeout ? 1 : 0;
  return v ? cudaMemsetAsync(p->status, 0, sizeof(int), s) : cudaSuccess;
}

void fluid_plan_destroy(FluidPlan *p) {
  if (p->tw) cudaFree(p->tw);
  if (p->lut) cudaFree(p->lut);
  if (p->spec) cudaFree(p->spec);
  if (p->status) cudaFree(p->status);
  if (p->any_tables) cudaFree(p->any_tables);
  delete p->any;
  std::memset(p, 0, sizeof(*p));
}

cudaError_t fluid_forward_field(const FluidPlan &p, const float *fx, const float *fy,
                                const float *fz, cudaStream_t s) {
  SrcField src{{fx, fy, fz}};
  if (p.fast) return fast_xy_forward(p, src, s);
  return any_forward(*p.any, src, p.split, s);
}

cudaError_t fluid_forward_force(const FluidPlan &p, const float *G, const float *A, int diff,
                                cudaStream_t s) {
  const SrcForce src = make_force(G, A, diff, p.sp);
  if (p.fast) return fast_xy_forward(p, src, s);
  return any_forward(*p.any, src, p.split, s);
}

cudaError_t fluid_forward_force_jac(const FluidPlan &p, const float *G, const float *A,
                                    const float *B, cudaStream_t s) {
  const SrcForce src = make_force(G, A, 2, p.sp, B);
  if (p.fast) return fast_xy_forward(p, src, s);
  return any_forward(*p.any, src, p.split, s);
}

cudaError_t fluid_solve(const FluidPlan &p, int inverse, cudaStream_t s) {
  if (p.fast) return fast_z_solve(p, inverse, s);
  return any_solve(*p.any, inverse, s);
}

cudaError_t fluid_inverse_store(const FluidPlan &p, float *ox, float *oy, float *oz,
                                cudaStream_t s) {
  DstField dst{{ox, oy, oz}};
  if (p.fast) return fast_xy_inverse(p, dst, s);
  return any_inverse(*p.any, dst, p.split, s);
}

cudaError_t fluid_inverse_compose(const FluidPlan &p, const ComposeArgs &a, cudaStream_t s) {
  if (!p.fast) return cudaErrorNotSupported;
  return fast_xy_inverse_compose(p, a, s);
}

cudaError_t fluid_inverse_store_neg(const FluidPlan &p, float *ox, float *oy, float *oz,
                                    cudaStream_t s) {
  DstNeg dst{{ox, oy, oz}};
  if (p.fast) return fast_xy_inverse(p, dst, s);
  return any_inverse(*p.any, dst, p.split, s);
}

cudaError_t fluid_inverse_axpby(const FluidPlan &p, float *vx, float *vy, float *vz,
                                const float *step, float sigma, cudaStream_t s) {
  DstAxpby dst{{vx, vy, vz}, step, sigma};
  if (p.fast) return fast_xy_inverse(p, dst, s);
  return any_inverse(*p.any, dst, p.split, s);
}

}  // namespace aw
