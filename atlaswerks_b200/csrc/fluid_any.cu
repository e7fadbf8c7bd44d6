// fluid_any.cu — the fluid operator's transforms for grids of any axis
// lengths, in place (the layout and the method: fluid_any.cuh).
//
//   xy forward   one block per (slab, component): the producer writes the
//                slab's row pairs as complex lines into shared memory, the x
//                and y stages run there, and one bulk copy takes the slab to
//                HBM as it lies.
//   z solve      one block per Q consecutive places of a slab, all three
//                components: the first radix is read from HBM straight into
//                registers, the last one, the 3 x 3 solve and the inverse's
//                first stay in registers (radices up to 5), and the
//                inverse's last goes back to HBM from registers: the tile
//                crosses shared memory four times in all for a length of two
//                factors.
//   xy inverse   the mirror of the forward pass, then the consumer.
//
// Every butterfly's lanes lie on consecutive lines (x), columns (y) or
// places (z), so a warp's twiddles are one broadcast and its data 16
// different banks: the x lines by the odd pitch, the columns by the order
// any_plan puts them in. Slabs beyond one block's shared memory run the same
// stages in an x and a y kernel with the slab in HBM between them.
#include <algorithm>
#include <climits>
#include <cmath>
#include <cstring>

#include "bulk.cuh"
#include "dft_reg.cuh"
#include "fluid.cuh"
#include "fluid_any.cuh"

namespace aw {

namespace {

constexpr int kXYMaxThreads = 768;  // 80 registers a thread: three blocks of 256 or one of 768 per SM
constexpr int kSplitMaxThreads = 512;  // 64 registers: 1024 threads per SM
constexpr int kZMaxThreads = 256;   // 64 registers: four blocks per SM

// exp(SIGN 2 pi i m / n) from the forward table
template <int SIGN>
AW_D float2 any_tw(const float2 *tw, int m) {
  const float2 w = tw[m];
  return SIGN < 0 ? w : make_float2(w.x, -w.y);
}

// One butterfly of a stage: reads get(r), writes put(k), both of r, k < R.
// Forward: DFT, then the twiddles; inverse: the twiddles, then the DFT.
template <int SIGN, int R, class Get, class Put>
AW_D void butterfly(const float2 *tw, int js, const Get &get, const Put &put) {
  float2 v[R];
#pragma unroll
  for (int r = 0; r < R; ++r) v[r] = get(r);
  if (SIGN > 0 && js) {
#pragma unroll
    for (int r = 1; r < R; ++r) v[r] = cmul(v[r], any_tw<SIGN>(tw, js * r));
  }
  dft<SIGN, R>(v);
  if (SIGN < 0 && js) {
#pragma unroll
    for (int r = 1; r < R; ++r) v[r] = cmul(v[r], any_tw<SIGN>(tw, js * r));
  }
#pragma unroll
  for (int r = 0; r < R; ++r) put(r, v[r]);
}

// f(integral constant R) for a butterfly radix
#define AW_RADIX(N, MAX) \
  case N: \
    if constexpr (N <= MAX) f(std::integral_constant<int, N>()); \
    break;
template <int RMAX, class F>
AW_D void with_radix(int R, const F &f) {
  switch (R) {
    AW_RADIX(2, RMAX)
    AW_RADIX(3, RMAX)
    AW_RADIX(4, RMAX)
    AW_RADIX(5, RMAX)
    AW_RADIX(6, RMAX)
    AW_RADIX(7, RMAX)
    AW_RADIX(8, RMAX)
    AW_RADIX(9, RMAX)
    AW_RADIX(10, RMAX)
    AW_RADIX(11, RMAX)
    AW_RADIX(12, RMAX)
    AW_RADIX(13, RMAX)
    AW_RADIX(14, RMAX)
    AW_RADIX(15, RMAX)
    AW_RADIX(16, RMAX)
  }
}
template <class F>
AW_D void with_even_radix(int R, const F &f) {
  switch (R) {
    AW_RADIX(2, kXYRadix)
    AW_RADIX(4, kXYRadix)
    AW_RADIX(6, kXYRadix)
    AW_RADIX(8, kXYRadix)
    AW_RADIX(10, kXYRadix)
    AW_RADIX(12, kXYRadix)
    AW_RADIX(14, kXYRadix)
    AW_RADIX(16, kXYRadix)
  }
}
static_assert(kSolveRadix == 5, "the radices of the fused z step");
template <class F>
AW_D void with_solve_radix(int R, const F &f) {
  switch (R) {
    AW_RADIX(2, kSolveRadix)
    AW_RADIX(3, kSolveRadix)
    AW_RADIX(4, kSolveRadix)
    AW_RADIX(5, kSolveRadix)
  }
}

// A stage of a prime radix above the registers', in place, by the whole
// block: a thread sums the results of kPrimeK pairs (k, R - k) of two
// butterflies in registers (over the pairs x[j] +- x[R-j], as dft<> does: 16
// multiply-adds to a twiddle pair read, its index stepped by k modulo n), and
// the block waits before any of the group's butterflies is written. kPrimeK:
// 4 in the slab kernels, 3 in the split and z kernels, by their registers. An
// axis of at most 512 has at most 64 chunks of k there and 85 here, and a
// block has the threads for them (128 and 256; a z block 64, and 256 from nz
// = 389 on, the first with more chunks, whose tile lets two share an SM).
template <int SIGN, int kPrimeK, class At>
AW_D void prime_stage(float2 *S, const float2 *tw, const AnyStage &st, int n, int nlines,
                      const IdxDiv &byLines, const At &at) {
  const int R = st.R, M = st.M, hh = (R - 1) / 2, nch = (hh + kPrimeK - 1) / kPrimeK;
  const int wr = n / R;  // table step of exp(-2 pi i / R)
  const int total = nlines * (n / R), half = (total + 1) / 2;
  const int G = blockDim.x / nch, g = threadIdx.x % G, ch = threadIdx.x / G;
  const int k0 = 1 + ch * kPrimeK;
  for (int base = 0; base < half; base += G) {
    const bool on = base + g < half && ch < nch;
    // Two butterflies, each of the stage's belonging to one thread of every
    // chunk: groups are not parted by a barrier, so a butterfly that another
    // group has too would be read after it was written. The thread of an odd
    // total's middle one takes it twice.
    const int bf[2] = {base + g, base + g + half < total ? base + g + half : base + g};
    float2 a[2][kPrimeK], b[2][kPrimeK], s[2];
    int w0[2], js[2], line[2];
    if (on) {
      int idx[kPrimeK];
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int bj = byLines.div(bf[e]);
        line[e] = bf[e] - bj * nlines;
        const int blk = st.byM.div(bj), j0 = bj - blk * M;
        w0[e] = blk * R * M + j0;
        js[e] = j0 * st.step;
        s[e] = S[at.of(line[e])(w0[e])];
      }
#pragma unroll
      for (int q = 0; q < kPrimeK; ++q) {
        idx[q] = 0;
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          a[e][q] = s[e];
          b[e][q] = make_float2(0.f, 0.f);
        }
      }
      const auto p0 = at.of(line[0]), p1 = at.of(line[1]);
      for (int j = 1; j <= hh; ++j) {
        float2 xa[2] = {S[p0(w0[0] + j * M)], S[p1(w0[1] + j * M)]};
        float2 xb[2] = {S[p0(w0[0] + (R - j) * M)], S[p1(w0[1] + (R - j) * M)]};
        float2 t[2], u[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          if (SIGN > 0 && M > 1) {
            xa[e] = cmul(xa[e], any_tw<SIGN>(tw, js[e] * j));
            xb[e] = cmul(xb[e], any_tw<SIGN>(tw, js[e] * (R - j)));
          }
          t[e] = cadd(xa[e], xb[e]);
          u[e] = csub(xa[e], xb[e]);
          s[e] = cadd(s[e], t[e]);
        }
#pragma unroll
        for (int q = 0; q < kPrimeK; ++q) {
          idx[q] += (k0 + q) * wr;  // k0 + q < R: one step back is enough
          if (idx[q] >= n) idx[q] -= n;
          const float2 w = any_tw<SIGN>(tw, idx[q]);
#pragma unroll
          for (int e = 0; e < 2; ++e) {
            a[e][q].x = fmaf(w.x, t[e].x, a[e][q].x);
            a[e][q].y = fmaf(w.x, t[e].y, a[e][q].y);
            b[e][q].x = fmaf(w.y, u[e].x, b[e][q].x);
            b[e][q].y = fmaf(w.y, u[e].y, b[e][q].y);
          }
        }
      }
    }
    __syncthreads();
    if (on) {
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const auto pl = at.of(line[e]);
        if (ch == 0) S[pl(w0[e])] = s[e];
#pragma unroll
        for (int q = 0; q < kPrimeK; ++q) {
          const int k = k0 + q;
          if (k > hh) break;
          float2 p = make_float2(a[e][q].x - b[e][q].y, a[e][q].y + b[e][q].x);
          float2 m = make_float2(a[e][q].x + b[e][q].y, a[e][q].y - b[e][q].x);
          if (SIGN < 0 && M > 1) {
            p = cmul(p, any_tw<SIGN>(tw, js[e] * k));
            m = cmul(m, any_tw<SIGN>(tw, js[e] * (R - k)));
          }
          S[pl(w0[e] + k * M)] = p;
          S[pl(w0[e] + (R - k) * M)] = m;
        }
      }
    }
  }
}

// One stage over nlines lines; at.of(line)(w) is the place of a line's value w
template <int SIGN, int RMAX, class At>
AW_D void line_stage(float2 *S, const float2 *tw, const AnyStage &st, int n, int nlines,
                     const IdxDiv &byLines, const At &at) {
  if (st.R > RMAX) {
    prime_stage<SIGN, (RMAX > 8 ? 4 : 3)>(S, tw, st, n, nlines, byLines, at);
    return;
  }
  with_radix<RMAX>(st.R, [&](auto rc) {
    constexpr int R = decltype(rc)::value;
    const int M = st.M, items = nlines * (n / R);
#pragma unroll 1
    for (int i = threadIdx.x; i < items; i += blockDim.x) {
      const int bj = byLines.div(i), line = i - bj * nlines;
      const int blk = st.byM.div(bj), j = bj - blk * M;
      const int w0 = blk * R * M + j;
      const auto pl = at.of(line);
      butterfly<SIGN, R>(
          tw, j * st.step, [&](int r) { return S[pl(w0 + r * M)]; },
          [&](int r, float2 v) { S[pl(w0 + r * M)] = v; });
    }
  });
}

struct LinePlace {
  int A, B, H, step;  // value w lies at w step + (w < H ? A : B)
  AW_D int operator()(int w) const { return w * step + (w < H ? A : B); }
};
// the lines of a slab: row pair p (x), or column c (y; B less the H lines
// that precede it). One type for both, so both run the same stage code.
struct AtSlab {
  const uint32_t *cols;  // null: x
  int H, pitch;
  AW_D LinePlace of(int l) const {
    if (!cols) return LinePlace{l * pitch, 0, INT_MAX, 1};
    const uint32_t ab = cols[l];
    return LinePlace{(int)(ab & 0xffffu), (int)(ab >> 16) - H * pitch, H, pitch};
  }
};
struct TilePlace {
  int base, q;
  AW_D int operator()(int w) const { return base + w * q; }
};
struct AtTile {  // tiles of n rows x q columns; line = c q + column of tile c
  int n, q, lq;
  AW_D TilePlace of(int l) const { return TilePlace{(l >> lq) * n * q + (l & (q - 1)), q}; }
};

AW_D void copy_table(float2 *dst, const float2 *src, int n) {
  for (int i = threadIdx.x; i < n; i += blockDim.x) dst[i] = __ldg(src + i);
}

// the two rows of one place pair of a column: X0 (row p) and X1 (row p + H)
AW_D void take_apart(const AnyXY &p, int c, float2 Z, float2 W, float2 &X0, float2 &X1) {
  if (c == 0) {  // the real columns 0 | nx / 2 (0 alone for odd nx)
    X0 = make_float2(Z.x, p.oddx ? 0.f : W.x);
    X1 = make_float2(Z.y, p.oddx ? 0.f : W.y);
  } else {
    X0 = make_float2(0.5f * (Z.x + W.x), 0.5f * (Z.y - W.y));
    X1 = make_float2(0.5f * (Z.y + W.y), -0.5f * (Z.x - W.x));
  }
}
AW_D void put_together(const AnyXY &p, int c, float2 X0, float2 X1, float2 &Z, float2 &W) {
  if (c == 0) {
    Z = make_float2(X0.x, X1.x);
    W = make_float2(X0.y, X1.y);
  } else {
    Z = make_float2(X0.x - X1.y, X0.y + X1.x);
    W = make_float2(X0.x + X1.y, X1.x - X0.y);
  }
}

// the packed column's rows ky and -ky: its sum column G, taken apart into
// column 0 at ky and column nx / 2 at ky
AW_D void unpack_pair(float2 G, float2 Gm, float2 &C0, float2 &CN) {
  C0 = make_float2(0.5f * (G.x + Gm.x), 0.5f * (G.y - Gm.y));
  CN = make_float2(0.5f * (G.y + Gm.y), -0.5f * (G.x - Gm.x));
}

// the producer's row pairs p0 .. p0 + np - 1 of slab z into S[0 ..], each a
// complex line; the places past nx zeroed. Consecutive threads take
// consecutive x, Src::kPairs row pairs each whose loads all go out before the
// first store.
template <class Src>
AW_D void produce(const AnyXY &p, const Src &src, float2 *S, int z, int comp, int p0, int np) {
  constexpr int U = Src::kPairs;
  const int nx = p.d.nx, total = np * nx;
  const auto in = src.at_slab(comp, z, p.H, p.d);
  for (int i0 = threadIdx.x; i0 < total; i0 += U * blockDim.x) {
    float2 v[U];
    int at[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      // past the end: the last item again (its loads are in range), not stored
      const int i = min(i0 + u * (int)blockDim.x, total - 1);
      const int l = p.byNx.div(i), x = i - l * nx;
      v[u] = in.pair(x, p0 + l);
      at[u] = l * p.pitch + x;
    }
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (i0 + u * (int)blockDim.x < total) S[at[u]] = v[u];
  }
  const int extra = p.pitch - nx;
  for (int i = threadIdx.x; i < np * extra; i += blockDim.x) {
    const int l = i / extra;
    S[l * p.pitch + nx + (i - l * extra)] = make_float2(0.f, 0.f);
  }
}

// the real rows of lines p0 .. p0 + np - 1 to the consumer
template <class Dst>
AW_D void consume(const AnyXY &p, const Dst &dst, const float2 *S, int z, int comp, int p0, int np) {
  constexpr int U = 4;
  const Dims d = p.d;
  const int nx = d.nx, total = np * nx;
  const auto out = dst.bind(comp);
  for (int i0 = threadIdx.x; i0 < total; i0 += U * blockDim.x) {
    if constexpr (Dst::kReads) {
      // every old value of the batch is read before any is written; an item
      // past the end or without a second row repeats the batch's first
      long idx[2 * U];
      float v[2 * U];
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int i = i0 + u * (int)blockDim.x;
        const int l = p.byNx.div(i < total ? i : i0), x = (i < total ? i : i0) - l * nx;
        const int y0 = p0 + l, y1 = y0 + p.H;
        const float2 Z = S[l * p.pitch + x];
        idx[2 * u] = i < total ? d.idx(x, y0, z) : -1;
        idx[2 * u + 1] = i < total && y1 < d.ny ? d.idx(x, y1, z) : -1;
        v[2 * u] = Z.x;
        v[2 * u + 1] = Z.y;
      }
      out.template store_some<2 * U>(idx, v);
    } else {
#pragma unroll
      for (int u = 0; u < U; ++u) {
        const int i = i0 + u * (int)blockDim.x;
        if (i >= total) break;
        const int l = p.byNx.div(i), x = i - l * nx;
        const int y0 = p0 + l, y1 = y0 + p.H;
        const float2 Z = S[l * p.pitch + x];
        out.store(d.idx(x, y0, z), Z.x);
        if (y1 < d.ny) out.store(d.idx(x, y1, z), Z.y);
      }
    }
  }
}

// ---- the slab kernels -------------------------------------------------------
template <class Src>
__global__ void __launch_bounds__(kXYMaxThreads) k_any_xy_fwd(const __grid_constant__ AnyXY p, Src src) {
  extern __shared__ __align__(128) float2 sm[];
  float2 *S = sm, *twx = S + p.slab, *twy = twx + p.x.n;
  uint32_t *cols = reinterpret_cast<uint32_t *>(twy + p.y.n);
  const int z = blockIdx.x, comp = blockIdx.y, H = p.H;
  copy_table(twx, p.x.tw, p.x.n);
  copy_table(twy, p.y.tw, p.y.n);
  for (int i = threadIdx.x; i < p.ncol; i += blockDim.x) cols[i] = __ldg(p.cols + i);
  if (threadIdx.x == 0 && (H * p.pitch & 1)) S[H * p.pitch] = make_float2(0.f, 0.f);
  wait_for_predecessors();
  produce(p, src, S, z, comp, 0, H);
  __syncthreads();
  // x and y stages by one loop, so that they share their code. Before the
  // y stages the rows are taken apart: with the first y stage (its radix
  // even: the rows r M + j and (r + R / 2) M + j are one line's pair), else
  // on their own.
#pragma unroll 1
  for (int s = 0; s < p.x.ns + p.y.ns; ++s) {
    const bool yy = s >= p.x.ns;
    const AnyLine &ln = yy ? p.y : p.x;
    if (s == p.x.ns) {
        if (p.fused) {
          const AnyStage st = p.y.st[0];
          with_even_radix(st.R, [&](auto rc) {
            constexpr int R = decltype(rc)::value;
            const int M = st.M, items = p.ncol * M;
#pragma unroll 1
            for (int i = threadIdx.x; i < items; i += blockDim.x) {
              const int j = p.byCol.div(i), c = i - j * p.ncol;
              const uint32_t ab = cols[c];
              float2 *A = S + j * p.pitch + (ab & 0xffffu), *B = S + j * p.pitch + (ab >> 16);
              const int row = M * p.pitch;
              float2 v[R];
#pragma unroll
              for (int r = 0; r < R / 2; ++r) take_apart(p, c, A[r * row], B[r * row], v[r], v[r + R / 2]);
              dft<-1, R>(v);
              if (j) {
#pragma unroll
                for (int r = 1; r < R; ++r) v[r] = cmul(v[r], twy[j * st.step * r]);
              }
#pragma unroll
              for (int r = 0; r < R / 2; ++r) {
                A[r * row] = v[r];
                B[r * row] = v[r + R / 2];
              }
            }
          });
        } else {
          for (int i = threadIdx.x; i < p.ncol * H; i += blockDim.x) {
            const int l = p.byCol.div(i), c = i - l * p.ncol;
            const uint32_t ab = cols[c];
            float2 *A = S + l * p.pitch + (ab & 0xffffu), *B = S + l * p.pitch + (ab >> 16);
            float2 X0, X1;
            take_apart(p, c, *A, *B, X0, X1);
            *A = X0;
            *B = X1;
          }
        }
      __syncthreads();
      if (p.fused) continue;
    }
    line_stage<-1, kXYRadix>(S, yy ? twy : twx, ln.st[yy ? s - p.x.ns : s], ln.n, yy ? p.ncol : H,
                   yy ? p.byCol : p.byH, AtSlab{yy ? cols : nullptr, H, p.pitch});
    __syncthreads();
  }
  const LinePlace at = AtSlab{cols, H, p.pitch}.of(0);
  for (int i = threadIdx.x; i < p.npk; i += blockDim.x) {
    const uint32_t ww = __ldg(p.packed + i);
    const int w = (int)(ww & 0xffffu), w2 = (int)(ww >> 16);
    float2 C0, CN;
    unpack_pair(S[at(w)], S[at(w2)], C0, CN);
    S[at(w)] = C0;
    // the first two pairs are their own (ky = 0, then ny / 2 of an even ny)
    S[w2 != w ? at(w2) : (i == 0 ? p.d.nx : p.pad1)] = CN;
  }
  dependents_may_start();
  fence_async_smem();
  __syncthreads();
  if (threadIdx.x == 0) {
    bulk_store(p.spec + ((long)comp * p.d.nz + z) * p.pcols, S, (uint32_t)(sizeof(float2) * p.slab));
    bulk_wait_read();
  }
}

template <class Dst>
__global__ void __launch_bounds__(kXYMaxThreads) k_any_xy_inv(const __grid_constant__ AnyXY p, Dst dst) {
  extern __shared__ __align__(128) float2 sm[];
  __shared__ uint64_t mbar;
  float2 *S = sm, *twx = S + p.slab, *twy = twx + p.x.n;
  uint32_t *cols = reinterpret_cast<uint32_t *>(twy + p.y.n);
  const int z = blockIdx.x, comp = blockIdx.y, H = p.H;
  copy_table(twx, p.x.tw, p.x.n);
  copy_table(twy, p.y.tw, p.y.n);
  for (int i = threadIdx.x; i < p.ncol; i += blockDim.x) cols[i] = __ldg(p.cols + i);
  wait_for_predecessors();
  if (threadIdx.x == 0) {
    const uint32_t bytes = (uint32_t)(sizeof(float2) * p.slab);
    mbar_init(&mbar, 1);
    mbar_expect_tx(&mbar, bytes);
    bulk_load(S, p.spec + ((long)comp * p.d.nz + z) * p.pcols, bytes, &mbar);
  }
  __syncthreads();
  // a slab that never lands: the status word says so and the block leaves as one
  if (__syncthreads_or(!mbar_wait(&mbar, 0, p.status))) return;
  const LinePlace at = AtSlab{cols, H, p.pitch}.of(0);
  for (int i = threadIdx.x; i < p.npk; i += blockDim.x) {
    const uint32_t ww = __ldg(p.packed + i);
    const int w = (int)(ww & 0xffffu), w2 = (int)(ww >> 16);
    const float2 a = S[at(w)];
    const float2 b = S[w2 != w ? at(w2) : (i == 0 ? p.d.nx : p.pad1)];
    S[at(w)] = make_float2(a.x - b.y, a.y + b.x);                      // C0 + i CN at ky
    if (w2 != w) S[at(w2)] = make_float2(a.x + b.y, b.x - a.y);        // and at -ky
  }
  __syncthreads();
  // the forward pass's loop, backwards
#pragma unroll 1
  for (int s = p.x.ns + p.y.ns - 1; s >= 0; --s) {
    const bool yy = s >= p.x.ns;
    const AnyLine &ln = yy ? p.y : p.x;
    if (s != p.x.ns || !p.fused) {
      line_stage<+1, kXYRadix>(S, yy ? twy : twx, ln.st[yy ? s - p.x.ns : s], ln.n, yy ? p.ncol : H,
                     yy ? p.byCol : p.byH, AtSlab{yy ? cols : nullptr, H, p.pitch});
      __syncthreads();
    }
    if (s == p.x.ns) {
        if (p.fused) {
          const AnyStage st = p.y.st[0];
          with_even_radix(st.R, [&](auto rc) {
            constexpr int R = decltype(rc)::value;
            const int M = st.M, items = p.ncol * M;
#pragma unroll 1
            for (int i = threadIdx.x; i < items; i += blockDim.x) {
              const int j = p.byCol.div(i), c = i - j * p.ncol;
              const uint32_t ab = cols[c];
              float2 *A = S + j * p.pitch + (ab & 0xffffu), *B = S + j * p.pitch + (ab >> 16);
              const int row = M * p.pitch;
              float2 v[R];
#pragma unroll
              for (int r = 0; r < R / 2; ++r) {
                v[r] = A[r * row];
                v[r + R / 2] = B[r * row];
              }
              if (j) {
#pragma unroll
                for (int r = 1; r < R; ++r) v[r] = cmul(v[r], any_tw<+1>(twy, j * st.step * r));
              }
              dft<+1, R>(v);
#pragma unroll
              for (int r = 0; r < R / 2; ++r) put_together(p, c, v[r], v[r + R / 2], A[r * row], B[r * row]);
            }
          });
        } else {
          for (int i = threadIdx.x; i < p.ncol * H; i += blockDim.x) {
            const int l = p.byCol.div(i), c = i - l * p.ncol;
            const uint32_t ab = cols[c];
            float2 *A = S + l * p.pitch + (ab & 0xffffu), *B = S + l * p.pitch + (ab >> 16);
            float2 Z, W;
            // an odd ny's last line has no second row
            const float2 X1 = l + H < p.d.ny ? *B : make_float2(0.f, 0.f);
            put_together(p, c, *A, X1, Z, W);
            *A = Z;
            *B = W;
          }
        }
      __syncthreads();
    }
  }
  consume(p, dst, S, z, comp, 0, H);
}

// ---- the split kernels: slabs larger than one block's shared memory ----------
// Radices up to 8 and 1024 threads on an SM, as in the z kernel: these passes
// wait for memory (x forward at 256 x 256 x 160: 71 us, with radices up to 16
// and 768 threads 86).
template <class Src>
__global__ void __launch_bounds__(kSplitMaxThreads, 2) k_any_x_fwd(const __grid_constant__ AnyXY p, Src src) {
  extern __shared__ __align__(128) float2 sm[];
  const int z = blockIdx.x, comp = blockIdx.y, p0 = blockIdx.z * p.P, np = min(p.P, p.H - p0);
  // the last batch takes the slab's odd place along
  const int places = np * p.pitch, whole = (places + 1) & ~1;
  float2 *S = sm, *twx = S + ((p.P * p.pitch + 1) & ~1);
  copy_table(twx, p.x.tw, p.x.n);
  if (threadIdx.x == 0 && whole > places) S[places] = make_float2(0.f, 0.f);
  wait_for_predecessors();
  produce(p, src, S, z, comp, p0, np);
  __syncthreads();
  const IdxDiv byL = np == p.P ? p.byP : p.byLast;
#pragma unroll 1
  for (int s = 0; s < p.x.ns; ++s) {
    line_stage<-1, kZRadix>(S, twx, p.x.st[s], p.x.n, np, byL, AtSlab{nullptr, 0, p.pitch});
    if (s + 1 == p.x.ns) fence_async_smem();
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    bulk_store(p.spec + ((long)comp * p.d.nz + z) * p.pcols + (long)p0 * p.pitch, S,
               (uint32_t)(sizeof(float2) * whole));
    bulk_wait_read();
  }
}

template <class Dst>
__global__ void __launch_bounds__(kSplitMaxThreads, 2) k_any_x_inv(const __grid_constant__ AnyXY p, Dst dst) {
  extern __shared__ __align__(128) float2 sm[];
  __shared__ uint64_t mbar;
  const int z = blockIdx.x, comp = blockIdx.y, p0 = blockIdx.z * p.P, np = min(p.P, p.H - p0);
  float2 *S = sm, *twx = S + ((p.P * p.pitch + 1) & ~1);
  copy_table(twx, p.x.tw, p.x.n);
  wait_for_predecessors();
  if (threadIdx.x == 0) {
    const uint32_t bytes = (uint32_t)(sizeof(float2) * ((np * p.pitch + 1) & ~1));
    mbar_init(&mbar, 1);
    mbar_expect_tx(&mbar, bytes);
    bulk_load(S, p.spec + ((long)comp * p.d.nz + z) * p.pcols + (long)p0 * p.pitch, bytes, &mbar);
  }
  __syncthreads();
  if (__syncthreads_or(!mbar_wait(&mbar, 0, p.status))) return;
  const IdxDiv byL = np == p.P ? p.byP : p.byLast;
#pragma unroll 1
  for (int s = p.x.ns - 1; s >= 0; --s) {
    line_stage<+1, kZRadix>(S, twx, p.x.st[s], p.x.n, np, byL, AtSlab{nullptr, 0, p.pitch});
    __syncthreads();
  }
  consume(p, dst, S, z, comp, p0, np);
}

// a batch of Q columns of one slab: rows taken apart into a [ny][Q] tile,
// the y stages, and back to the columns' places (SIGN > 0: the mirror)
template <int SIGN>
__global__ void __launch_bounds__(kSplitMaxThreads, 2) k_any_y(const __grid_constant__ AnyXY p) {
  extern __shared__ __align__(128) float2 sm[];
  const int Q = p.Q, lq = 31 - __clz(Q), ny = p.d.ny, H = p.H;
  float2 *T = sm, *twy = T + ny * Q;
  const int c0 = blockIdx.z * Q, nc = min(Q, p.ncol - c0);
  float2 *C = p.spec + ((long)blockIdx.y * p.d.nz + blockIdx.x) * p.pcols;
  copy_table(twy, p.y.tw, ny);
  const int q = threadIdx.x & (Q - 1);
  const uint32_t ab = __ldg(p.cols + c0 + min(q, nc - 1));
  const int A = (int)(ab & 0xffffu), B = (int)(ab >> 16);
  const int rows = (int)blockDim.x >> lq, r0 = (int)threadIdx.x >> lq;
  const AtTile at{ny, Q, lq};
  wait_for_predecessors();
  if (SIGN < 0) {
#pragma unroll 4
    for (int l = r0; l < H; l += rows) {
      const float2 Z = C[(long)l * p.pitch + A], W = C[(long)l * p.pitch + B];
      float2 X0, X1;
      take_apart(p, c0 + q, Z, W, X0, X1);
      T[l * Q + q] = X0;
      if (l + H < ny) T[(l + H) * Q + q] = X1;
    }
  } else {
#pragma unroll 4
    for (int l = r0; l < H; l += rows) {
      const float2 a = C[(long)l * p.pitch + A], b = C[(long)l * p.pitch + B];
      T[l * Q + q] = a;
      if (l + H < ny) T[(l + H) * Q + q] = b;
    }
  }
  __syncthreads();
  if (SIGN > 0 && c0 == 0) {
    for (int i = threadIdx.x; i < p.npk; i += blockDim.x) {
      const uint32_t ww = __ldg(p.packed + i);
      const int w = (int)(ww & 0xffffu), w2 = (int)(ww >> 16);
      const float2 a = T[w * Q], b = w2 != w ? T[w2 * Q] : C[i == 0 ? p.d.nx : p.pad1];
      T[w * Q] = make_float2(a.x - b.y, a.y + b.x);
      if (w2 != w) T[w2 * Q] = make_float2(a.x + b.y, b.x - a.y);
    }
    __syncthreads();
  }
#pragma unroll 1
  for (int s = 0; s < p.y.ns; ++s) {
    line_stage<SIGN, kZRadix>(T, twy, p.y.st[SIGN < 0 ? s : p.y.ns - 1 - s], ny, Q, p.byQ, at);
    __syncthreads();
  }
  if (SIGN < 0 && c0 == 0) {
    for (int i = threadIdx.x; i < p.npk; i += blockDim.x) {
      const uint32_t ww = __ldg(p.packed + i);
      const int w = (int)(ww & 0xffffu), w2 = (int)(ww >> 16);
      float2 C0, CN;
      unpack_pair(T[w * Q], T[w2 * Q], C0, CN);
      T[w * Q] = C0;
      if (w2 != w)
        T[w2 * Q] = CN;
      else
        C[i == 0 ? p.d.nx : p.pad1] = CN;
    }
    __syncthreads();
  }
  if (q < nc) {
    for (int l = r0; l < H; l += rows) {
      float2 Z = T[l * Q + q], W = l + H < ny ? T[(l + H) * Q + q] : make_float2(0.f, 0.f);
      if (SIGN > 0) {
        const float2 X0 = Z, X1 = W;
        put_together(p, c0 + q, X0, X1, Z, W);
      }
      C[(long)l * p.pitch + A] = Z;
      C[(long)l * p.pitch + B] = W;
    }
  }
}

// ---- z ----------------------------------------------------------------------
// L = diag(D) + beta s s^T with D_i = lambda + beta e_i, e = (1 - cos)^2 / sp^2
// (L_ii = lambda - beta c_i and c = (2 cos - 2) / sp^2, so -c_i - s_i^2 = e_i;
// DiffOper.cxx:590-639, 1005-1116): all of D is positive, and the inverse is
// the rank-one update D^-1 - beta D^-1 s s^T D^-1 / (1 + beta s^T D^-1 s)
// (Sherman & Morrison 1950), with no cancellation in forming D and no square
// root. Each divisor has a division of its own: 1 / (D0 D1) and one more
// product would save two of the four (z pass 84.1 against 86.9 us at 180 x 216
// x 180, 105.6 against 108.5 at 256 x 256 x 160), but leave the range of a
// float for diagonal terms beyond 1e19 or below 1e-19.
struct ZSolve {
  float sx, sy, ex, ey, lxy;  // of the column; lxy = gamma - alpha (cx + cy)
  float alpha, beta, invN;
  int inverse;
  AW_D void operator()(const float4 &lz, float2 &a, float2 &b, float2 &c) const {
    const float lambda = lxy - alpha * lz.x, sz = lz.y;
    const float d0 = lambda + beta * ex, d1 = lambda + beta * ey, d2 = lambda + beta * lz.z;
    if (inverse) {
      const float r0 = 1.0f / d0, r1 = 1.0f / d1, r2 = 1.0f / d2;
      const float u0 = r0 * sx, u1 = r1 * sy, u2 = r2 * sz;
      const float g = beta / (1.0f + beta * (u0 * sx + u1 * sy + u2 * sz));
      const float tx = g * (u0 * a.x + u1 * b.x + u2 * c.x), ty = g * (u0 * a.y + u1 * b.y + u2 * c.y);
      a = make_float2((r0 * a.x - u0 * tx) * invN, (r0 * a.y - u0 * ty) * invN);
      b = make_float2((r1 * b.x - u1 * tx) * invN, (r1 * b.y - u1 * ty) * invN);
      c = make_float2((r2 * c.x - u2 * tx) * invN, (r2 * c.y - u2 * ty) * invN);
    } else {
      const float tx = beta * (sx * a.x + sy * b.x + sz * c.x), ty = beta * (sx * a.y + sy * b.y + sz * c.y);
      a = make_float2((d0 * a.x + sx * tx) * invN, (d0 * a.y + sx * ty) * invN);
      b = make_float2((d1 * b.x + sy * tx) * invN, (d1 * b.y + sy * ty) * invN);
      c = make_float2((d2 * c.x + sz * tx) * invN, (d2 * c.y + sz * ty) * invN);
    }
  }
};

__global__ void __launch_bounds__(kZMaxThreads, 4) k_any_z(const __grid_constant__ AnyZ p, int inverse) {
  extern __shared__ __align__(128) float2 sm[];
  const int nz = p.d.nz, Q = p.q, lq = p.lq, tile = nz * Q, ns = p.z.ns;
  float4 *lz = reinterpret_cast<float4 *>(sm);  // first: 16-byte values
  float2 *T = reinterpret_cast<float2 *>(lz + nz), *tw = T + 3 * tile;
  copy_table(tw, p.z.tw, nz);
  for (int i = threadIdx.x; i < nz; i += blockDim.x) lz[i] = __ldg(p.lutz + i);
  const int q = threadIdx.x & (Q - 1);
  const long col = (long)blockIdx.x * Q + q;
  float2 *G = p.spec + col;
  // pcols is a multiple of 16: a tile of 32 may reach past it
  const bool on = col < p.pcols;
  ZSolve solve;
  {
    const uint32_t k = __ldg(p.kxy + (on ? col : 0));
    const float4 a = __ldg(p.lutx + (k & 0xffffu)), b = __ldg(p.luty + (k >> 16));
    solve = ZSolve{a.y, b.y, a.z, b.z, p.gamma - p.alpha * (a.x + b.x), p.alpha, p.beta, p.invN, inverse};
  }
  const AtTile at{nz, Q, lq};
  const AnyStage first = p.z.st[0];
  const int rows = (int)blockDim.x >> lq, r0 = (int)threadIdx.x >> lq;
  wait_for_predecessors();
  __syncthreads();
  // the first radix straight from HBM (a single stage: a plain copy)
  const bool direct = ns > 1 && first.R <= kZRadix;
  if (direct) {
    with_radix<kZRadix>(first.R, [&](auto rc) {
      constexpr int R = decltype(rc)::value;
      const int M = first.M;
#pragma unroll 1
      for (int i = r0; i < 3 * M; i += rows) {
        const int c = i >= 2 * M ? 2 : (i >= M ? 1 : 0), j = i - c * M;
        const float2 *g = G + ((long)c * nz + j) * p.pcols;
        float2 *t = T + (c * nz + j) * Q + q;
        if (on)
          butterfly<-1, R>(
              tw, j * first.step, [&](int r) { return g[(long)r * M * p.pcols]; },
              [&](int r, float2 v) { t[r * M * Q] = v; });
      }
    });
  } else {
#pragma unroll 4
    for (int i = r0; i < 3 * nz; i += rows)
      T[i * Q + q] = on ? G[(long)i * p.pcols] : make_float2(0.f, 0.f);
  }
  __syncthreads();
  const int s0 = direct ? 1 : 0, s1 = p.fused ? ns - 1 : ns;
#pragma unroll 1
  for (int s = s0; s < s1; ++s) {
    line_stage<-1, kZRadix>(T, tw, p.z.st[s], nz, 3 * Q, p.by3Q, at);
    __syncthreads();
  }
  if (p.fused) {
    with_solve_radix(p.z.st[ns - 1].R, [&](auto rc) {
      constexpr int R = decltype(rc)::value;
      const int nb = nz / R;
#pragma unroll 1
      for (int b = r0; b < nb; b += rows) {
        float2 *t = T + b * R * Q + q;
        float2 v[3][R];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
#pragma unroll
          for (int r = 0; r < R; ++r) v[c][r] = t[c * tile + r * Q];
          dft<-1, R>(v[c]);
        }
#pragma unroll
        for (int r = 0; r < R; ++r) solve(lz[b * R + r], v[0][r], v[1][r], v[2][r]);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
          dft<+1, R>(v[c]);
#pragma unroll
          for (int r = 0; r < R; ++r) t[c * tile + r * Q] = v[c][r];
        }
      }
    });
  } else {
    for (int w = r0; w < nz; w += rows) {
      float2 *t = T + w * Q + q;
      solve(lz[w], t[0], t[tile], t[2 * tile]);
    }
  }
  dependents_may_start();
  __syncthreads();
#pragma unroll 1
  for (int s = s1 - 1; s >= s0; --s) {
    line_stage<+1, kZRadix>(T, tw, p.z.st[s], nz, 3 * Q, p.by3Q, at);
    __syncthreads();
  }
  if (!on) return;
  if (direct) {
    with_radix<kZRadix>(first.R, [&](auto rc) {
      constexpr int R = decltype(rc)::value;
      const int M = first.M;
#pragma unroll 1
      for (int i = r0; i < 3 * M; i += rows) {
        const int c = i >= 2 * M ? 2 : (i >= M ? 1 : 0), j = i - c * M;
        float2 *g = G + ((long)c * nz + j) * p.pcols;
        const float2 *t = T + (c * nz + j) * Q + q;
        butterfly<+1, R>(
            tw, j * first.step, [&](int r) { return t[r * M * Q]; },
            [&](int r, float2 v) { g[(long)r * M * p.pcols] = v; });
      }
    });
  } else {
    for (int i = r0; i < 3 * nz; i += rows) G[(long)i * p.pcols] = T[i * Q + q];
  }
}

// ---- plans --------------------------------------------------------------------
// The fewest radices of at most rmax whose product is n (primes above it as
// they are, last), the smallest sum among those; first even when
// even_first and n is even; the last at most last_max. False: no such list
// within kAnyStages.
bool split_smooth(int n, int parts, bool first, bool even_first, int rmax, int last_max,
                  std::vector<int> &cur, std::vector<int> &best, int &best_sum, int sum) {
  if (parts == 1) {
    if (n < 2 || n > rmax || n > last_max || (first && even_first && n % 2)) return false;
    if (sum + n < best_sum) {
      best_sum = sum + n;
      best = cur;
      best.push_back(n);
    }
    return true;
  }
  bool any = false;
  for (int r = rmax; r >= 2; --r) {
    if (n % r || (first && even_first && r % 2)) continue;
    cur.push_back(r);
    any = split_smooth(n / r, parts - 1, false, even_first, rmax, last_max, cur, best, best_sum,
                       sum + r) || any;
    cur.pop_back();
  }
  return any;
}

bool any_radices(int n, bool even_first, int rmax, int last_max, std::vector<int> &out) {
  std::vector<int> primes;
  int m = n;
  for (int p = 2; p <= rmax; ++p)
    while (m % p == 0) m /= p;
  const int smooth = n / m;
  for (int p = rmax + 1; m > 1; ++p)
    while (m % p == 0) {
      primes.push_back(p);
      m /= p;
    }
  out.clear();
  if (!primes.empty()) last_max = rmax;
  if (smooth > 1) {
    for (int parts = 1; parts <= kAnyStages && out.empty(); ++parts) {
      std::vector<int> cur, best;
      int sum = 1 << 30;
      if (split_smooth(smooth, parts, true, even_first && smooth % 2 == 0, rmax, last_max, cur, best,
                       sum, 0))
        out = best;
    }
    if (out.empty()) {
      // no list ends in a small enough radix (a 7 alone)
      return last_max < rmax && any_radices(n, even_first, rmax, rmax, out);
    }
  }
  out.insert(out.end(), primes.begin(), primes.end());
  return (int)out.size() <= kAnyStages;
}

void fill_line(AnyLine *l, int n, const std::vector<int> &rad) {
  l->n = n;
  l->ns = (int)rad.size();
  int Ns = n;
  for (int s = 0; s < l->ns; ++s) {
    const int R = rad[s], M = Ns / R;
    l->st[s] = AnyStage{R, M, n / Ns, make_idxdiv((uint32_t)M)};
    Ns = M;
  }
}

std::vector<int> position_freq(int n, const std::vector<int> &rad) {
  std::vector<int> f(n);
  for (int p = 0; p < n; ++p) {
    int k = 0, mul = 1, rem = p, N = n;
    for (int R : rad) {
      const int M = N / R, dg = rem / M;
      rem %= M;
      k += dg * mul;
      mul *= R;
      N = M;
    }
    f[p] = k;
  }
  return f;
}

void fill_symbols(int n, double sp, std::vector<float4> &out) {
  out.resize(n);
  const double s = 2.0 * M_PI / (double)n;
  for (int k = 0; k < n; ++k) {
    const double co = std::cos(s * k);
    out[k] = make_float4((float)((2.0 * co - 2.0) / (sp * sp)), (float)(std::sin(s * k) / sp),
                         (float)((1.0 - co) * (1.0 - co) / (sp * sp)), 0.f);
  }
}

}  // namespace

bool any_plan(AnyPlan *p, AnyTables *t, const Dims &d, const Spacing &sp, float alpha, float beta,
              float gamma, bool split) {
  std::vector<int> rx, ry, rz;
  const int rmax = split ? kZRadix : kXYRadix;
  if (!any_radices(d.nx, false, rmax, rmax, rx) || !any_radices(d.ny, true, rmax, rmax, ry) ||
      !any_radices(d.nz, false, kZRadix, kSolveRadix, rz))
    return false;
  AnyXY &a = p->xy;
  a.d = d;
  const int nx = d.nx, ny = d.ny, H = (ny + 1) / 2;
  a.H = H;
  a.oddx = nx & 1;
  a.pitch = nx + 1 + a.oddx;
  if (a.pitch % 2 == 0) ++a.pitch;
  if (H == 1 && !a.oddx) a.pitch += 2;  // both extra places on the one line
  a.pad1 = H > 1 ? a.pitch + nx : nx + 1;
  a.slab = (H * a.pitch + 1) & ~1;
  a.pcols = (a.slab + 15) / 16 * 16;
  fill_line(&a.x, nx, rx);
  fill_line(&a.y, ny, ry);
  a.fused = ny % 2 == 0 && ry[0] % 2 == 0 && ry[0] <= kXYRadix && !split;
  a.byNx = make_idxdiv((uint32_t)nx);
  a.byH = make_idxdiv((uint32_t)H);
  const std::vector<int> fx = position_freq(nx, rx), fy = position_freq(ny, ry);
  std::vector<int> px(nx), py(ny);
  for (int i = 0; i < nx; ++i) px[fx[i]] = i;
  for (int i = 0; i < ny; ++i) py[fy[i]] = i;
  // columns (A, B, kx): the packed one first
  struct Col {
    int A, B, k;
  };
  std::vector<Col> cols{{px[0], a.oddx ? nx : px[nx / 2], 0}}, rest;
  for (int k = 1; k < (nx + 1) / 2; ++k) rest.push_back({px[k], px[nx - k], k});
  std::sort(rest.begin(), rest.end(), [](const Col &u, const Col &v) { return u.A < v.A; });
  if (split) {
    // the first radix's block k0 of a line mirrors onto block R0 - k0: the
    // columns of such a pair of blocks together, so that a batch of them
    // covers two whole runs of places in HBM
    const int run = nx / rx[0];
    auto lower = [&](const Col &c) { return std::min(c.A / run, c.B / run); };
    for (Col &c : rest)
      if (c.B / run < c.A / run) c = Col{c.B, c.A, nx - c.k};
    std::sort(rest.begin(), rest.end(), [&](const Col &u, const Col &v) {
      return lower(u) != lower(v) ? lower(u) < lower(v) : u.A < v.A;
    });
    cols.insert(cols.end(), rest.begin(), rest.end());
  } else {
    // 16 columns in a row (a half warp's) on 16 banks at A and at B, as far
    // as they can be: the first that fits, either end of it as A
    while (!rest.empty()) {
      const size_t g = cols.size() / 16 * 16;
      unsigned ua = 0, ub = 0;
      for (size_t i = g; i < cols.size(); ++i) {
        ua |= 1u << (cols[i].A & 15);
        ub |= 1u << (cols[i].B & 15);
      }
      size_t pick = 0;
      bool swap = false;
      int best = 3;
      for (size_t i = 0; i < rest.size() && best; ++i)
        for (int w = 0; w < 2 && best; ++w) {
          const int A = w ? rest[i].B : rest[i].A, B = w ? rest[i].A : rest[i].B;
          const int cost = ((ua >> (A & 15)) & 1) + ((ub >> (B & 15)) & 1);
          if (cost < best) {
            best = cost;
            pick = i;
            swap = w != 0;
          }
        }
      const Col c = rest[pick];
      rest.erase(rest.begin() + (long)pick);
      cols.push_back(swap ? Col{c.B, c.A, nx - c.k} : c);
    }
  }
  a.ncol = (int)cols.size();
  a.byCol = make_idxdiv((uint32_t)a.ncol);
  auto at = [&](const Col &c, int w) { return w < H ? w * a.pitch + c.A : (w - H) * a.pitch + c.B; };
  t->kxy.assign(a.pcols, 0);
  for (const Col &c : cols)
    for (int w = 0; w < ny; ++w) t->kxy[at(c, w)] = (uint32_t)c.k | (uint32_t)fy[w] << 16;
  t->packed.clear();
  if (!a.oddx) {
    // the self-paired rows first (their second places are the extra ones)
    for (int self = 1; self >= 0; --self)
      for (int ky = 0; ky <= ny / 2; ++ky) {
        const int w = py[ky], w2 = py[(ny - ky) % ny];
        if ((w == w2) != (self == 1)) continue;
        const int second = w != w2 ? at(cols[0], w2) : (t->packed.empty() ? nx : a.pad1);
        t->kxy[at(cols[0], w)] = (uint32_t)ky << 16;
        t->kxy[second] = (uint32_t)(nx / 2) | (uint32_t)ky << 16;
        t->packed.push_back((uint32_t)w | (uint32_t)w2 << 16);
      }
  }
  a.npk = (int)t->packed.size();
  t->cols.clear();
  for (const Col &c : cols) t->cols.push_back((uint32_t)c.A | (uint32_t)c.B << 16);

  AnyZ &z = p->z;
  z.d = d;
  z.pcols = a.pcols;
  fill_line(&z.z, d.nz, rz);
  z.fused = rz.back() <= kSolveRadix;
  z.alpha = alpha;
  z.beta = beta;
  z.gamma = gamma;
  z.invN = 1.0f / (float)d.n();
  fill_symbols(nx, sp.x, t->lutx);
  fill_symbols(ny, sp.y, t->luty);
  std::vector<float4> lz;
  fill_symbols(d.nz, sp.z, lz);
  const std::vector<int> fz = position_freq(d.nz, rz);
  t->lutz.resize(d.nz);
  for (int i = 0; i < d.nz; ++i) t->lutz[i] = lz[fz[i]];
  return true;
}

size_t any_smem_xy(const AnyXY &a) {
  return sizeof(float2) * ((size_t)a.slab + a.x.n + a.y.n) + sizeof(uint32_t) * a.ncol;
}

// the z pass's columns per block and its threads
void any_set_z(AnyPlan *p, int q) {
  p->z.q = q;
  p->z.lq = 0;
  while ((1 << p->z.lq) < q) ++p->z.lq;
  p->z.by3Q = make_idxdiv((uint32_t)(3 * q));
  p->smem_z = sizeof(float2) * (3 * (size_t)p->z.d.nz * q + p->z.d.nz) + sizeof(float4) * p->z.d.nz;
}

// shared memory of the split path's y pass with Q columns per block
size_t any_smem_y(const AnyXY &a, int Q) { return sizeof(float2) * ((size_t)a.d.ny * Q + a.d.ny); }

// the split path's row pairs (rounded up to even: a batch starts on 16
// bytes) and columns (up to a power of two of at most 64 whose tile fits)
// per block
void any_set_split(AnyPlan *p, int P, int Q, size_t maxsm) {
  AnyXY &a = p->xy;
  a.P = (P + 1) & ~1;
  a.byP = make_idxdiv((uint32_t)a.P);
  const int last = a.H - (a.H - 1) / a.P * a.P;
  a.byLast = make_idxdiv((uint32_t)last);
  a.Q = 1;
  while (a.Q < Q && a.Q < 64 && any_smem_y(a, 2 * a.Q) <= maxsm) a.Q *= 2;
  a.byQ = make_idxdiv((uint32_t)a.Q);
  p->smem_x = sizeof(float2) * ((((size_t)a.P * a.pitch + 1) & ~(size_t)1) + a.x.n);
  p->smem_y = any_smem_y(a, a.Q);
  p->threads_y = a.Q >= 32 ? 512 : 256;
}

template <class Src>
cudaError_t any_forward(const AnyPlan &p, const Src &src, bool split, cudaStream_t s) {
  const AnyXY &a = p.xy;
  if (!split)
    return launched(
        launch_early(k_any_xy_fwd<Src>, dim3(a.d.nz, 3), p.threads_xy, p.smem_xy, s, a, src));
  const cudaError_t e = launch_early(k_any_x_fwd<Src>, dim3(a.d.nz, 3, (a.H + a.P - 1) / a.P), 256,
                                     p.smem_x, s, a, src);
  if (e != cudaSuccess) return launched(e);
  return launched(launch_early(k_any_y<-1>, dim3(a.d.nz, 3, (a.ncol + a.Q - 1) / a.Q), p.threads_y,
                               p.smem_y, s, a));
}

template <class Dst>
cudaError_t any_inverse(const AnyPlan &p, const Dst &dst, bool split, cudaStream_t s) {
  const AnyXY &a = p.xy;
  if (!split)
    return launched(
        launch_early(k_any_xy_inv<Dst>, dim3(a.d.nz, 3), p.threads_xy, p.smem_xy, s, a, dst));
  const cudaError_t e = launch_early(k_any_y<+1>, dim3(a.d.nz, 3, (a.ncol + a.Q - 1) / a.Q),
                                     p.threads_y, p.smem_y, s, a);
  if (e != cudaSuccess) return launched(e);
  return launched(launch_early(k_any_x_inv<Dst>, dim3(a.d.nz, 3, (a.H + a.P - 1) / a.P), 256, p.smem_x,
                               s, a, dst));
}

cudaError_t any_solve(const AnyPlan &p, int inverse, cudaStream_t s) {
  const int grid = (int)((p.z.pcols + p.z.q - 1) / p.z.q);
  return launched(launch_early(k_any_z, dim3(grid), p.threads_z, p.smem_z, s, p.z, inverse));
}

// the kernels of a plan and the shared memory each needs
std::vector<std::pair<const void *, size_t>> any_kernels(const AnyPlan &p, bool split) {
  std::vector<std::pair<const void *, size_t>> k{{(const void *)k_any_z, p.smem_z}};
  auto add = [&](const void *f, size_t b) { k.emplace_back(f, b); };
  if (split) {
    add((const void *)k_any_x_fwd<SrcField>, p.smem_x);
    add((const void *)k_any_x_fwd<SrcForce>, p.smem_x);
    add((const void *)k_any_x_inv<DstField>, p.smem_x);
    add((const void *)k_any_x_inv<DstAxpby>, p.smem_x);
    add((const void *)k_any_x_inv<DstNeg>, p.smem_x);
    add((const void *)k_any_y<-1>, p.smem_y);
    add((const void *)k_any_y<+1>, p.smem_y);
  } else {
    add((const void *)k_any_xy_fwd<SrcField>, p.smem_xy);
    add((const void *)k_any_xy_fwd<SrcForce>, p.smem_xy);
    add((const void *)k_any_xy_inv<DstField>, p.smem_xy);
    add((const void *)k_any_xy_inv<DstAxpby>, p.smem_xy);
    add((const void *)k_any_xy_inv<DstNeg>, p.smem_xy);
  }
  return k;
}

template cudaError_t any_forward<SrcField>(const AnyPlan &, const SrcField &, bool, cudaStream_t);
template cudaError_t any_forward<SrcForce>(const AnyPlan &, const SrcForce &, bool, cudaStream_t);
template cudaError_t any_inverse<DstField>(const AnyPlan &, const DstField &, bool, cudaStream_t);
template cudaError_t any_inverse<DstAxpby>(const AnyPlan &, const DstAxpby &, bool, cudaStream_t);
template cudaError_t any_inverse<DstNeg>(const AnyPlan &, const DstNeg &, bool, cudaStream_t);

}  // namespace aw
