// splat.cu — deterministic counting-sort splat (see splat.cuh).
#include <algorithm>
#include <climits>

#include "splat.cuh"

namespace aw {

namespace {

constexpr int kScanThreads = 256;
constexpr int kScanItems = 4;
constexpr int kScanBlock = kScanThreads * kScanItems;

inline size_t align256(size_t b) { return (b + 255) & ~size_t(255); }

// bucket of a source: the cell of its h, shifted by one so that
// h in (-1, 0) lands in bucket 0. Returns -1 for sources the reference
// skips: those outside the volume grown by one voxel
// (HField3DUtils.txx:1110-1112).
AW_D long bucket_of(const Dims &d, float px, float py, float pz) {
  if (!(px > -1.0f && px < (float)d.nx && py > -1.0f && py < (float)d.ny && pz > -1.0f &&
        pz < (float)d.nz))
    return -1;
  int fx, fy, fz;
  float gx, gy, gz;
  cell_of(px, py, pz, fx, fy, fz, gx, gy, gz);
  return ((long)(fz + 1) * (d.ny + 1) + (fy + 1)) * (d.nx + 1) + (fx + 1);
}

// bucket sizes, and every source's place in its bucket (in arrival order)
__global__ void __launch_bounds__(kRowThreads)
    k_count(const float *__restrict__ hx, const float *__restrict__ hy, const float *__restrict__ hz,
            Dims d, int *__restrict__ counts, int *__restrict__ place) {
  early_entry();
  Voxel v;
  if (!voxel_of(d, v)) return;
  const long b = bucket_of(d, hx[v.i], hy[v.i], hz[v.i]);
  if (b >= 0) place[v.i] = atomicAdd(counts + b, 1);
}

// block-local exclusive scan of kScanBlock ints held 4 per thread
AW_D int block_scan(int (&a)[kScanItems], int *wsum) {
  int tsum = 0;
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    const int x = a[k];
    a[k] = tsum;
    tsum += x;
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int incl = tsum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  if (lane == 31) wsum[warp] = incl;
  __syncthreads();
  if (warp == 0) {
    int w = lane < kScanThreads / 32 ? wsum[lane] : 0;
    int wi = w;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, wi, o);
      if (lane >= o) wi += y;
    }
    if (lane < kScanThreads / 32) wsum[lane] = wi - w;  // exclusive warp offsets
    if (lane == kScanThreads / 32 - 1) wsum[kScanThreads / 32] = wi;  // block total
  }
  __syncthreads();
  const int base = wsum[warp] + (incl - tsum);
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) a[k] += base;
  const int total = wsum[kScanThreads / 32];
  __syncthreads();
  return total;
}

__global__ void __launch_bounds__(kScanThreads)
    k_scan_reduce(const int *__restrict__ x, long n, int *__restrict__ blocksums) {
  early_entry();
  const long b0 = (long)blockIdx.x * kScanBlock;
  int s = 0;
  for (int k = 0; k < kScanItems; ++k) {
    const long i = b0 + (long)k * kScanThreads + threadIdx.x;
    if (i < n) s += x[i];
  }
  __shared__ int ws[kScanThreads / 32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    int t = 0;
    for (int w = 0; w < kScanThreads / 32; ++w) t += ws[w];
    blocksums[blockIdx.x] = t;
  }
}

// one block: exclusive scan of the block sums, chunk by chunk
__global__ void __launch_bounds__(kScanThreads) k_scan_blocksums(int *__restrict__ bs, int nb) {
  early_entry();
  __shared__ int wsum[kScanThreads / 32 + 1];
  int carry = 0;
  for (int c0 = 0; c0 < nb; c0 += kScanBlock) {
    int a[kScanItems];
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
      const int i = c0 + threadIdx.x * kScanItems + k;
      a[k] = i < nb ? bs[i] : 0;
    }
    const int total = block_scan(a, wsum);
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
      const int i = c0 + threadIdx.x * kScanItems + k;
      if (i < nb) bs[i] = a[k] + carry;
    }
    carry += total;
    __syncthreads();
  }
}

// exclusive scan in place; x[n] receives the total. SUM: blocksums holds the
// blocks' own sums, and each block adds up those before it (up to kScanSum of
// them: a 16 KB read from L2 against a launch of its own for their scan).
constexpr int kScanSum = 4096;
template <bool SUM>
__global__ void __launch_bounds__(kScanThreads)
    k_scan_apply(int *__restrict__ x, long n, const int *__restrict__ blocksums) {
  early_entry();
  __shared__ int wsum[kScanThreads / 32 + 1];
  const long b0 = (long)blockIdx.x * kScanBlock;
  int a[kScanItems];
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    const long i = b0 + (long)threadIdx.x * kScanItems + k;
    a[k] = i < n ? x[i] : 0;
  }
  const int total = block_scan(a, wsum);
  int off = 0;
  if (SUM) {
    for (int j = threadIdx.x; j < (int)blockIdx.x; j += kScanThreads) off += blocksums[j];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) off += __shfl_xor_sync(0xffffffffu, off, o);
    __syncthreads();  // block_scan's use of wsum is over
    if ((threadIdx.x & 31) == 0) wsum[threadIdx.x >> 5] = off;
    __syncthreads();
    off = 0;
#pragma unroll
    for (int w = 0; w < kScanThreads / 32; ++w) off += wsum[w];
  } else {
    off = blocksums[blockIdx.x];
  }
#pragma unroll
  for (int k = 0; k < kScanItems; ++k) {
    const long i = b0 + (long)threadIdx.x * kScanItems + k;
    if (i < n) x[i] = a[k] + off;
  }
  if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) x[n] = off + total;
}

// weight of corner (cx, cy, cz) of a source with fractions r, rounded to
// float as forwardApply writes it (HField3DUtils.txx:1116-1123): the product
// runs left to right, in double once a (1.0 - r) factor has entered it and
// in float before, so w110 = (rx*ry in float) * (1.0 - rz) and w111 =
// rx*ry*rz in float.
struct Fractions {
  float rx, ry, rz;
};
AW_D Fractions fractions_of(float px, float py, float pz) {
  int fx, fy, fz;
  float gx, gy, gz;
  cell_of(px, py, pz, fx, fy, fz, gx, gy, gz);
  return Fractions{fsub(px, gx), fsub(py, gy), fsub(pz, gz)};
}
AW_D float corner_weight(const Fractions &f, int cx, int cy, int cz) {
  if (cx && cy) {
    const float rxy = fmul(f.rx, f.ry);
    return cz ? fmul(rxy, f.rz) : __double2float_rn(dmul((double)rxy, dsub(1.0, (double)f.rz)));
  }
  const double ax = cx ? (double)f.rx : dsub(1.0, (double)f.rx);
  const double ay = cy ? (double)f.ry : dsub(1.0, (double)f.ry);
  const double az = cz ? (double)f.rz : dsub(1.0, (double)f.rz);
  return __double2float_rn(dmul(dmul(ax, ay), az));
}

// sources to their buckets, in arrival order
__global__ void __launch_bounds__(kRowThreads)
    k_scatter(const float *__restrict__ hx, const float *__restrict__ hy,
              const float *__restrict__ hz, Dims d, const int *__restrict__ offsets,
              const int *__restrict__ place, int *__restrict__ order) {
  early_entry();
  Voxel v;
  if (!voxel_of(d, v)) return;
  const long b = bucket_of(d, hx[v.i], hy[v.i], hz[v.i]);
  if (b >= 0) order[offsets[b] + place[v.i]] = (int)v.i;
}

// Buckets of up to kSmallBucket sources are insertion-sorted by one thread
// (at most k(k-1)/2 moves); longer ones, which only a strongly compressing
// or collapsed map produces, by the whole CTA with a stable radix sort.
constexpr int kSortThreads = 256;
constexpr int kSortWarps = kSortThreads / 32;
constexpr int kSmallBucket = 64;

struct SortShared {
  int large[kSortThreads];         // block-local indices of the long buckets
  int nlarge;
  int base[256];                   // running digit offsets within the segment
  int wc[kSortWarps][256];         // per-warp digit counts of one 256-key tile
  int red[2][kSortWarps];
};

// Stable LSD radix sort of the distinct source indices order[s, e) by the
// whole CTA, 8 bits a pass over the keys' range, ping-ponging through
// tmp[s, e). Every key's position comes from counts (no atomic order), so
// the result is the ascending order whatever the input order; the work is
// O(k) per pass and at most four passes.
AW_D void block_radix_sort(int *__restrict__ order, int *__restrict__ tmp, int s, int e,
                           SortShared &sh) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int mn = INT_MAX, mx = INT_MIN;
  for (int i = s + tid; i < e; i += kSortThreads) {
    const int k = order[i];
    mn = min(mn, k);
    mx = max(mx, k);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    mn = min(mn, __shfl_xor_sync(0xffffffffu, mn, o));
    mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  }
  if (lane == 0) {
    sh.red[0][warp] = mn;
    sh.red[1][warp] = mx;
  }
  __syncthreads();
  mn = sh.red[0][0];
  mx = sh.red[1][0];
  for (int w = 1; w < kSortWarps; ++w) {
    mn = min(mn, sh.red[0][w]);
    mx = max(mx, sh.red[1][w]);
  }
  __syncthreads();
  const unsigned range = (unsigned)mx - (unsigned)mn;
  const int passes = range ? (32 - __clz((int)range) + 7) / 8 : 0;
  int *src = order, *dst = tmp;
  const unsigned lt = (1u << lane) - 1u;
  for (int p = 0; p < passes; ++p) {
    const int shift = 8 * p;
    sh.base[tid] = 0;
    __syncthreads();
    for (int i = s + tid; i < e; i += kSortThreads)
      atomicAdd(&sh.base[(((unsigned)src[i] - (unsigned)mn) >> shift) & 255u], 1);
    __syncthreads();
    {  // exclusive scan of the 256 digit counts, one per thread
      const int c = sh.base[tid];
      int incl = c;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += y;
      }
      if (lane == 31) sh.red[0][warp] = incl;
      __syncthreads();
      int off = 0;
      for (int w = 0; w < warp; ++w) off += sh.red[0][w];
      sh.base[tid] = off + incl - c;
      __syncthreads();
    }
    for (int t0 = s; t0 < e; t0 += kSortThreads) {
      const int i = t0 + tid;
      const bool valid = i < e;
      const int key = valid ? src[i] : 0;
      const int dg = valid ? (int)((((unsigned)key - (unsigned)mn) >> shift) & 255u) : 256;
#pragma unroll
      for (int w = 0; w < kSortWarps; ++w) sh.wc[w][tid] = 0;
      __syncthreads();
      const unsigned peers = __match_any_sync(0xffffffffu, dg);
      if (valid && (__ffs(peers) - 1) == lane) sh.wc[warp][dg] = __popc(peers);
      __syncthreads();
      if (valid) {
        int pre = sh.base[dg];
        for (int w = 0; w < warp; ++w) pre += sh.wc[w][dg];
        dst[s + pre + __popc(peers & lt)] = key;
      }
      __syncthreads();
      int add = 0;
#pragma unroll
      for (int w = 0; w < kSortWarps; ++w) add += sh.wc[w][tid];
      sh.base[tid] += add;
      __syncthreads();
    }
    int *t = src;
    src = dst;
    dst = t;
  }
  if (src != order) {
    for (int i = s + tid; i < e; i += kSortThreads) order[i] = src[i];
  }
  __syncthreads();
}

// Sorts every bucket by source index. One CTA per 256 buckets; tmp (the
// sources' places, dead by now) holds at least n + 2 ints.
__global__ void __launch_bounds__(kSortThreads)
    k_bucket_sort(const int *__restrict__ offsets, int *__restrict__ order, int *__restrict__ tmp,
                  long next, long n) {
  early_entry();
  __shared__ SortShared sh;
  // the sums' queue (tmp's first n places, then its count and the blocks
  // done with it) starts empty
  if (blockIdx.x == 0 && threadIdx.x < 2) tmp[n + threadIdx.x] = 0;
  const long b = (long)blockIdx.x * kSortThreads + threadIdx.x;
  const int s = b < next ? offsets[b] : 0, e = b < next ? offsets[b + 1] : 0;
  const bool large = e - s > kSmallBucket;
  if (!large) {
    for (int i = s + 1; i < e; ++i) {
      const int key = order[i];
      int j = i - 1;
      while (j >= s && order[j] > key) {
        order[j + 1] = order[j];
        --j;
      }
      order[j + 1] = key;
    }
  }
  if (!__syncthreads_or(large)) return;
  if (threadIdx.x == 0) sh.nlarge = 0;
  __syncthreads();
  if (large) sh.large[atomicAdd(&sh.nlarge, 1)] = threadIdx.x;
  __syncthreads();
  const int nl = sh.nlarge;
  for (int q = 0; q < nl; ++q) {
    const long bb = (long)blockIdx.x * kSortThreads + sh.large[q];
    block_radix_sort(order, tmp, offsets[bb], offsets[bb + 1], sh);
  }
}

// A source's eight contributions, corner weight times value, at its place in
// the order: one plane of n per corner (dx + 2 dy + 4 dz), so that the sums
// of neighbouring destinations, which want the same corner of neighbouring
// places, read consecutive values, one load a contribution and none that
// waits for the source's index.
__global__ void __launch_bounds__(256)
    k_products(const int *__restrict__ order, const int *__restrict__ total, long n,
               const float *__restrict__ img, const float *__restrict__ hx,
               const float *__restrict__ hy, const float *__restrict__ hz,
               float *__restrict__ prod) {
  early_entry();
  const int p = blockIdx.x * 256 + threadIdx.x;
  if (p >= *total) return;
  const int m = order[p];
  const Fractions f = fractions_of(__ldg(hx + m), __ldg(hy + m), __ldg(hz + m));
  const float v = __ldg(img + m);
#pragma unroll
  for (int k = 0; k < 8; ++k)
    prod[k * n + p] = fmul(corner_weight(f, k & 1, (k >> 1) & 1, (k >> 2) & 1), v);
}

// Every destination sums its contributions in source order, the order
// forwardApply adds them. Its candidates lie in eight buckets: the cell
// v - (dx, dy, dz) contributes its corner (dx, dy, dz). Buckets dx = 1 and
// dx = 0 of one (dy, dz) are adjacent in the order, so three offsets bound
// both, and four such ranges hold all candidates, eight on average.
//
// Most destinations meet their sources in order when the ranges are walked
// from (dy, dz) = (1, 1) down to (0, 0): up to kPer candidates of each range
// are fetched at once, their indices and their products (k_products), and
// where the indices rise, the products are added as they come. The others, 14 % of
// them on a map with half a voxel of relief and 35 % on a compressing one,
// lie scattered over nearly every warp: k_gather only queues them, and
// k_gather_queued takes them one per thread, so that whole warps do the
// ordering instead of a few lanes of each. There each pair of candidates out
// of order moves its two ranks apart, kept four bits each in two words (a
// compare and an addition a pair, without divergence), and the products go
// to shared memory by rank and are added from there. A destination with more
// than kMore candidates beyond the first kPer of their ranges merges its
// eight sorted buckets one source at a time.
constexpr int kGatherThreads = 256, kQueuedThreads = 128;
constexpr int kPer = 3, kMore = 4, kFirst = 4 * kPer, kSlots = kFirst + kMore;
static_assert(kSlots == 16, "ranks of four bits in two words");

struct GatherArgs {
  Dims d;
  long n;
  IdxDiv byNx, byNy;
  const float *img, *hx, *hy, *hz;
  const float *prod;  // PRE: the products; else they are formed here
  const int *offsets, *order;
  int *queue;  // n destinations, then their count and the blocks done with it
  float *out;
  float bg;
};

// the four candidate ranges of a destination, each [beg, mid) at dx = 1 and
// [mid, end) at dx = 0
struct Ranges {
  int beg[4], mid[4], end[4];  // sum_by_merging indexes them in this order
};
AW_D Ranges ranges_of(const GatherArgs &a, int i) {
  const int row = a.byNx.div(i), x = i - row * a.d.nx, z = a.byNy.div(row), y = row - z * a.d.ny;
  const int sy = a.d.nx + 1, sz = sy * (a.d.ny + 1);  // buckets fit 31 bits
  Ranges q;
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int dy = r & 1, dz = r >> 1;
    const int *o = a.offsets + ((z - dz + 1) * sz + (y - dy + 1) * sy + x);
    q.beg[r] = __ldg(o);
    q.mid[r] = __ldg(o + 1);
    q.end[r] = __ldg(o + 2);
  }
  return q;
}
// the product of source m at place p of the order; corner k = dx + 2 dy + 4 dz
template <bool PRE>
AW_D float contribution(const GatherArgs &a, int p, int m, int k) {
  if (PRE) return __ldg(a.prod + ((long)k * a.n + p));
  return fmul(corner_weight(fractions_of(__ldg(a.hx + m), __ldg(a.hy + m), __ldg(a.hz + m)), k & 1,
                            (k >> 1) & 1, (k >> 2) & 1),
              __ldg(a.img + m));
}

// Any number of candidates: the smallest head of the eight sorted buckets,
// one source a step, the same instructions whichever bucket it is. Heads
// carry their bucket in the low bits (source * 8 + bucket; grids of 2^29
// voxels and more compare for it), so the smallest names it, and the thread's
// column of the ranks' shared memory holds each bucket's place and the head
// behind. What a step fetches, the element two behind and the contribution,
// the next one takes, so that neither is waited for. A splat at 128^3, against
// eight compares with a branch and its loads a step: 4.6 sources a cell 446 ->
// 384 us (with noise 506 -> 391), 64 a cell 934 -> 809, 512 sources on one
// place 983 -> 642.
template <bool PRE>
__device__ __noinline__ float sum_by_merging(const GatherArgs &a, const Ranges &q, int *place,
                                             unsigned *behind) {
  constexpr unsigned kNone = 0xffffffffu;
  const bool tagged = a.n < (1L << 29);
  auto head = [&](int p, int e, int k) {
    if (p >= e) return kNone;
    const unsigned m = (unsigned)__ldg(a.order + p);
    return tagged ? m * 8 + k : m;
  };
  unsigned cur[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    const int p = (k & 1) ? q.beg[k >> 1] : q.mid[k >> 1];
    const int e = (k & 1) ? q.mid[k >> 1] : q.end[k >> 1];
    place[k * kQueuedThreads] = p;
    cur[k] = head(p, e, k);
    behind[k * kQueuedThreads] = head(p + 1, e, k);
  }
  const int *const bounds = reinterpret_cast<const int *>(&q);  // beg, mid, end
  float acc = a.bg, held = 0.f;
  int from = -1;             // the last step's bucket,
  unsigned fetched = kNone;  // and the head that it fetched
  while (true) {
    const unsigned key = min(min(min(cur[0], cur[1]), min(cur[2], cur[3])),
                             min(min(cur[4], cur[5]), min(cur[6], cur[7])));
    if (from >= 0) {
      acc = fadd(acc, held);
      behind[from * kQueuedThreads] = fetched;
    }
    if (key == kNone) return acc;
    int sel = (int)(key & 7u), m = (int)(key >> 3);
    if (!tagged) {
      m = (int)key;
#pragma unroll
      for (int k = 0; k < 8; ++k) sel = cur[k] == key ? k : sel;  // a source lies in one bucket
    }
    const int at = place[sel * kQueuedThreads];
    const unsigned next = behind[sel * kQueuedThreads];
    place[sel * kQueuedThreads] = at + 1;
    held = contribution<PRE>(a, at, m, sel);
    fetched = head(at + 2, bounds[(sel >> 1) + ((sel & 1) ? 4 : 8)], sel);
    from = sel;
#pragma unroll
    for (int k = 0; k < 8; ++k) cur[k] = cur[k] == key ? next : cur[k];
  }
}

// candidate c of the first kPer of every range, in the walk's order: its
// range, and its index or INT_MAX
AW_D constexpr int range_of(int c) { return 3 - c / kPer; }
AW_D void first_candidates(const GatherArgs &a, const Ranges &q, int *m) {
#pragma unroll
  for (int r = 3; r >= 0; --r) {
    const int *o = a.order + q.beg[r];
    const int len = q.end[r] - q.beg[r];
#pragma unroll
    for (int c = 0; c < kPer; ++c) m[(3 - r) * kPer + c] = c < len ? __ldg(o + c) : INT_MAX;
  }
}
// their products (0 for none)
template <bool PRE>
AW_D void first_products(const GatherArgs &a, const Ranges &q, const int *m, float *pr) {
#pragma unroll
  for (int r = 3; r >= 0; --r) {
    // corner dx = 0 of range r, and dx = 1 one plane on
    const float *w0 = PRE ? a.prod + ((long)(2 * r) * a.n + q.beg[r]) : nullptr;
    const float *w1 = PRE ? w0 + a.n : nullptr;
    const int len = q.end[r] - q.beg[r], ones = q.mid[r] - q.beg[r];
#pragma unroll
    for (int c = 0; c < kPer; ++c) {
      const int i = (3 - r) * kPer + c;
      if (PRE)
        pr[i] = c < len ? __ldg((c < ones ? w1 : w0) + c) : 0.f;
      else
        pr[i] = c < len ? contribution<PRE>(a, q.beg[r] + c, m[i], 2 * r + (c < ones ? 1 : 0)) : 0.f;
    }
  }
}

template <bool PRE>
__global__ void __launch_bounds__(kGatherThreads) k_gather(const __grid_constant__ GatherArgs a) {
  early_entry();
  const int i = blockIdx.x * kGatherThreads + threadIdx.x;
  bool later = false;
  if (i < a.n) {
    Ranges q = ranges_of(a, i);
    int m[kFirst], top = -1;
    float pr[kFirst];
    // a range of more candidates than are fetched here: nothing is fetched
#pragma unroll
    for (int r = 0; r < 4; ++r) later = later || q.end[r] - q.beg[r] > kPer;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      q.mid[r] = later ? q.beg[r] : q.mid[r];
      q.end[r] = later ? q.beg[r] : q.end[r];
    }
    first_candidates(a, q, m);
    if (PRE) first_products<PRE>(a, q, m, pr);
#pragma unroll
    for (int r = 3; r >= 0; --r) {
      const int *c = m + (3 - r) * kPer;
      static_assert(kPer == 3, "a range's largest index");
      const int len = q.end[r] - q.beg[r];
      later = later || c[0] < top || c[1] < c[0] || c[2] < c[1];
      top = max(top, len > 2 ? c[2] : (len > 1 ? c[1] : (len > 0 ? c[0] : -1)));
    }
    if (!later) {
      float acc = a.bg;
      if (!PRE) first_products<PRE>(a, q, m, pr);
#pragma unroll
      for (int c = 0; c < kFirst; ++c)
        if (m[c] != INT_MAX) acc = fadd(acc, pr[c]);
      a.out[i] = acc;
    }
  }
  const unsigned who = __ballot_sync(0xffffffffu, later);
  if (!who) return;
  const int lane = threadIdx.x & 31;
  int at = 0;
  if (lane == 0) at = atomicAdd(a.queue + a.n, __popc(who));
  at = __shfl_sync(0xffffffffu, at, 0);
  if (later) a.queue[at + __popc(who & ((1u << lane) - 1u))] = i;
}

// entries i < j of the walk: out of order, their ranks move apart
AW_D void rank_pair(unsigned (&rk)[2], const int *m, int i, int j) {
  if (m[j] >= m[i]) return;
  if (i / 8 == j / 8) {
    rk[i / 8] += (1u << (4 * (i % 8))) - (1u << (4 * (j % 8)));
  } else {
    rk[i / 8] += 1u << (4 * (i % 8));
    rk[j / 8] -= 1u << (4 * (j % 8));
  }
}

// the queued destinations, one per thread; the last block to finish empties
// the queue for the next image splatted by the same map
template <bool PRE>
__global__ void __launch_bounds__(kQueuedThreads) k_gather_queued(const __grid_constant__ GatherArgs a) {
  early_entry();
  __shared__ float byrank[kSlots][kQueuedThreads];
  const int tid = threadIdx.x, count = *(volatile int *)(a.queue + a.n);
  for (int t = blockIdx.x * kQueuedThreads + tid; t < count; t += gridDim.x * kQueuedThreads) {
    const int i = a.queue[t];
    const Ranges q = ranges_of(a, i);
    int more = 0, total = 0;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int len = q.end[r] - q.beg[r];
      more += max(len - kPer, 0);
      total += len;
    }
    // where a quarter of the warp is such destinations, all of it merges: the
    // others' lists are shorter, and ordering them first would come on top (a
    // regular scaling by 0.75 at 128^3 389 -> 369 us; by a single one, LDMM's
    // maps take 0.5 % longer)
    const bool merge = more > kMore;
    const bool many = __popc(__ballot_sync(__activemask(), merge)) >= 8;
    if (merge || many) {
      a.out[i] = sum_by_merging<PRE>(a, q, reinterpret_cast<int *>(&byrank[0][tid]),
                                     reinterpret_cast<unsigned *>(&byrank[8][tid]));
      continue;
    }
    int m[kSlots];
    float pr[kSlots];
    first_candidates(a, q, m);
    first_products<PRE>(a, q, m, pr);
    // ranks start as the walk's own order; the absent sort behind
    unsigned rk[2] = {0x76543210u, 0xfedcba98u};
#pragma unroll
    for (int j = 1; j < kFirst; ++j)
#pragma unroll
      for (int c = 0; c < j; ++c) rank_pair(rk, m, c, j);
    if (more) {
      // the c-th candidate past the first kPer of its range, ranges in the
      // walk's order
#pragma unroll
      for (int c = 0; c < kMore; ++c) {
        int left = c, p = -1, k = 0;
#pragma unroll
        for (int r = 3; r >= 0; --r) {
          const int over = max(q.end[r] - q.beg[r] - kPer, 0);
          if (p < 0 && left < over) {
            p = q.beg[r] + kPer + left;
            k = (p < q.mid[r] ? 1 : 0) + 2 * r;
          }
          left -= over;
        }
        m[kFirst + c] = p >= 0 ? __ldg(a.order + p) : INT_MAX;
        pr[kFirst + c] = p >= 0 ? contribution<PRE>(a, p, m[kFirst + c], k) : 0.f;
      }
#pragma unroll
      for (int j = kFirst; j < kSlots; ++j)
#pragma unroll
        for (int c = 0; c < j; ++c) rank_pair(rk, m, c, j);
#pragma unroll
      for (int c = kFirst; c < kSlots; ++c) byrank[(rk[1] >> (4 * (c % 8))) & 15u][tid] = pr[c];
    }
#pragma unroll
    for (int c = 0; c < kFirst; ++c) byrank[(rk[c / 8] >> (4 * (c % 8))) & 15u][tid] = pr[c];
    float acc = a.bg;
    for (int c = 0; c < total; ++c) acc = fadd(acc, byrank[c][tid]);
    a.out[i] = acc;
  }
  __syncthreads();
  if (tid == 0) {
    unsigned *done = reinterpret_cast<unsigned *>(a.queue + a.n + 1);
    if (atomicInc(done, gridDim.x - 1) == gridDim.x - 1) a.queue[a.n] = 0;
  }
}

}  // namespace

size_t splat_scratch_bytes(const Dims &d, bool products) {
  const long next = (long)(d.nx + 1) * (d.ny + 1) * (d.nz + 1);
  const long nb = (next + kScanBlock - 1) / kScanBlock;
  return align256(sizeof(int) * (next + 1)) + align256(sizeof(int) * next) +
         align256(sizeof(int) * d.n()) + align256(sizeof(int) * nb) +
         (products ? align256(sizeof(float) * 8 * d.n()) : 0);
}

void splat_work_bind(SplatWork *w, const Dims &d, void *scratch, bool products) {
  char *p = static_cast<char *>(scratch);
  w->d = d;
  w->next = (long)(d.nx + 1) * (d.ny + 1) * (d.nz + 1);
  w->nblocks = (int)((w->next + kScanBlock - 1) / kScanBlock);
  w->offsets = reinterpret_cast<int *>(p);
  p += align256(sizeof(int) * (w->next + 1));
  w->cursor = reinterpret_cast<int *>(p);
  p += align256(sizeof(int) * w->next);
  w->order = reinterpret_cast<int *>(p);
  p += align256(sizeof(int) * d.n());
  w->blocksums = reinterpret_cast<int *>(p);
  p += align256(sizeof(int) * w->nblocks);
  w->prod = products ? reinterpret_cast<float *>(p) : nullptr;
  int dev = 0;
  w->sms = 148;
  if (cudaGetDevice(&dev) == cudaSuccess)
    cudaDeviceGetAttribute(&w->sms, cudaDevAttrMultiProcessorCount, dev);
}

cudaError_t splat_sort(const SplatWork &w, const float *hx, const float *hy, const float *hz,
                       cudaStream_t s) {
  const Dims d = w.d;
  cudaError_t e;
  if ((e = cudaMemsetAsync(w.offsets, 0, sizeof(int) * (w.next + 1), s)) != cudaSuccess) return e;
  launch_early(k_count, row_grid(d), kRowThreads, 0, s, hx, hy, hz, d, w.offsets, w.cursor);
  launch_early(k_scan_reduce, dim3(w.nblocks), kScanThreads, 0, s, w.offsets, w.next, w.blocksums);
  if (w.nblocks <= kScanSum) {
    launch_early(k_scan_apply<true>, dim3(w.nblocks), kScanThreads, 0, s, w.offsets, w.next,
                 w.blocksums);
  } else {
    launch_early(k_scan_blocksums, dim3(1), kScanThreads, 0, s, w.blocksums, w.nblocks);
    launch_early(k_scan_apply<false>, dim3(w.nblocks), kScanThreads, 0, s, w.offsets, w.next,
                 w.blocksums);
  }
  launch_early(k_scatter, row_grid(d), kRowThreads, 0, s, hx, hy, hz, d, w.offsets, w.cursor,
               w.order);
  launch_early(k_bucket_sort, dim3((int)((w.next + kSortThreads - 1) / kSortThreads)), kSortThreads,
               0, s, w.offsets, w.order, w.cursor, w.next, d.n());
  return cudaGetLastError();
}

cudaError_t splat_gather(const SplatWork &w, const float *img, const float *hx, const float *hy,
                         const float *hz, float *out, float bg, cudaStream_t s) {
  const Dims d = w.d;
  const GatherArgs a{d,  d.n(), make_idxdiv((uint32_t)d.nx), make_idxdiv((uint32_t)d.ny), img, hx, hy,
                     hz, w.prod, w.offsets, w.order, w.cursor, out, bg};
  const unsigned grid = (unsigned)((d.n() + kGatherThreads - 1) / kGatherThreads);
  // seven blocks an SM, or one thread per destination
  const unsigned queued = (unsigned)std::min<long>((d.n() + kQueuedThreads - 1) / kQueuedThreads, 7L * w.sms);
  if (w.prod) {
    launch_early(k_products, dim3((unsigned)((d.n() + 255) / 256)), 256, 0, s, w.order,
                 w.offsets + w.next, d.n(), img, hx, hy, hz, w.prod);
    launch_early(k_gather<true>, dim3(grid), kGatherThreads, 0, s, a);
    launch_early(k_gather_queued<true>, dim3(queued), kQueuedThreads, 0, s, a);
  } else {
    launch_early(k_gather<false>, dim3(grid), kGatherThreads, 0, s, a);
    launch_early(k_gather_queued<false>, dim3(queued), kQueuedThreads, 0, s, a);
  }
  return cudaGetLastError();
}

cudaError_t splat(const SplatWork &w, const float *img, const float *hx, const float *hy,
                  const float *hz, float *out, float bg, cudaStream_t s) {
  const cudaError_t e = splat_sort(w, hx, hy, hz, s);
  return e != cudaSuccess ? e : splat_gather(w, img, hx, hy, hz, out, bg, s);
}

}  // namespace aw
