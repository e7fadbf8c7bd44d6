// fluid_any.cuh — the in-place transforms of the fluid operator for any grid
// (fluid_any.cu), and the tables they run from.
//
// A line of n values is transformed in place, stage by stage: a butterfly
// of radix R reads R values a stride apart and writes its results to the
// same R places (decimation in frequency forward, its mirror inverse).
// Nothing is reordered: position p of a transformed line holds frequency
// freq(p), the digits of p reversed, and the pointwise solve between the
// forward and the inverse transform looks its frequencies up by position.
//
// One (z, component) slab, as the xy kernels hold it in shared memory and as
// it lies in HBM between the passes:
//   H = ceil(ny / 2) lines of `pitch` complex places (pitch odd). Line p
//   first holds the rows p and p + H of the real field as real and
//   imaginary part. After the x transform the values at places A (kx) and
//   B (nx - kx) of line p give column kx of the half spectrum of both rows,
//   X0 = (Z[A] + conj Z[B]) / 2 and X1 = (Z[A] - conj Z[B]) / 2i, which
//   take the two places: row w of column (A, B) lies at
//     w < H ? (w, A) : (w - H, B).
//   Columns kx = 0 and nx / 2 of an even nx are real, share one complex
//   column through the y transform, and are then taken apart into the
//   places of ky and -ky (column 0 at ky, column nx / 2 at the place of
//   -ky: the other half of each follows by symmetry); their two self-paired
//   rows need one more place each, the slots past nx of lines 0 and 1.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <utility>
#include <vector>

#include "aw_common.cuh"

namespace aw {

constexpr int kAnyStages = 6;   // 512 = 8 x 8 x 8; 343 = 7 x 7 x 7
// Butterflies in registers: up to 16 in the xy kernels, whose stages are
// parted by barriers of the whole block (fewer stages win: the inverse slab
// kernel at 128^3 takes 25.3 us with radices up to 16, 30.0 with up to 8),
// up to 8 in the z kernel and 5 in its fused step, where more threads and
// less code win (22.1 against 26.3 us with 16 and 10: half of the stalls
// there were for instructions). Larger primes are summed by the block.
constexpr int kXYRadix = 16, kZRadix = 8, kSolveRadix = 5;

struct AnyStage {
  int R, M;      // radix, and the stride of its inputs (the sub-length after it)
  int step;      // twiddle table step: exp(-2 pi i j k / (R M)) = tw[j k step]
  IdxDiv byM;
};
struct AnyLine {
  int n, ns;
  AnyStage st[kAnyStages];
  const float2 *tw;
};

struct AnyXY {
  Dims d;
  int H, pitch, slab;  // lines, places per line, places per slab (even)
  int ncol, oddx, fused;  // columns; nx odd; ny even: the first y stage takes the rows apart
  int npk;             // row pairs (ky, -ky) of the packed column (0: nx odd)
  int pad1;            // the second extra place (the first is nx)
  AnyLine x, y;
  IdxDiv byH, byNx, byCol;
  const uint32_t *cols;   // [ncol] A | B << 16, the packed column first
  const uint32_t *packed; // [npk] place w | w' << 16 of ky, -ky
  float2 *spec;
  long pcols;          // places per slab in HBM (a multiple of 16)
  int *status;
  // the split path's batches
  int P, Q;
  IdxDiv byP, byLast, byQ;
};

struct AnyZ {
  Dims d;
  long pcols;
  int q, lq;           // columns per block, a power of two, and its log2
  IdxDiv by3Q;
  AnyLine z;
  int fused;           // the last radix is at most kSolveRadix
  const uint32_t *kxy; // [pcols] kx | ky << 16
  const float4 *lutx, *luty, *lutz;  // c, s, e of a frequency (lutz by position)
  float alpha, beta, gamma, invN;
  float2 *spec;
};

struct AnyPlan {
  AnyXY xy;
  AnyZ z;
  int threads_xy, threads_y, threads_z;
  size_t smem_xy, smem_x, smem_y, smem_z;
};

// Host tables of a grid's plan; fluid_plan_create uploads them
struct AnyTables {
  std::vector<uint32_t> cols, packed, kxy;
  std::vector<float4> lutx, luty, lutz;
};

// Fills the plan (all but the device pointers and the launch shapes) and
// its tables. False when an axis needs more than kAnyStages stages.
bool any_plan(AnyPlan *p, AnyTables *t, const Dims &d, const Spacing &sp, float alpha, float beta,
              float gamma, bool split);
size_t any_smem_xy(const AnyXY &a);
size_t any_smem_y(const AnyXY &a, int Q);
void any_set_z(AnyPlan *p, int q);
void any_set_split(AnyPlan *p, int P, int Q, size_t maxsm);
// the kernels of a plan and the shared memory each needs
std::vector<std::pair<const void *, size_t>> any_kernels(const AnyPlan &p, bool split);

template <class Src>
cudaError_t any_forward(const AnyPlan &p, const Src &src, bool split, cudaStream_t s);
template <class Dst>
cudaError_t any_inverse(const AnyPlan &p, const Dst &dst, bool split, cudaStream_t s);
cudaError_t any_solve(const AnyPlan &p, int inverse, cudaStream_t s);

}  // namespace aw
