// splat.cuh — deterministic splatting (the adjoint of trilinear
// interpolation), HField3DUtils::forwardApply with normalize = false
// (UtilitiesDataTypes/HField3DUtils.txx:1058-1279).
//
// The reference CPU adds each source voxel's eight weighted corner
// contributions in source (z, y, x) order, in float; the reference GPU path
// uses int32 fixed-point atomics (CUDACommon/src/cudaSplatAtomic.cu:379-448).
// Here the sources are bucketed by the cell their h lands in (counting sort:
// count, exclusive scan, scatter, per-bucket sort by source index), their
// eight contributions are formed once each, and every destination voxel adds
// those of the eight buckets that can reach it sequentially in source-index
// order (how it finds that order depends on their number, splat.cu). No float
// atomics, run-to-run bitwise identical, and with identical inputs bitwise
// equal to the reference CPU.
#pragma once

#include "aw_common.cuh"

namespace aw {

// device scratch of one splat, sized for a grid (extended by one cell per
// axis for sources landing in (-1, 0))
struct SplatWork {
  Dims d;
  long next;        // (nx+1)(ny+1)(nz+1)
  int *offsets;     // next + 1: bucket counts, then exclusive offsets
  int *cursor;      // next: each source's place in its bucket, the sort's scratch, the sums' queue
  int *order;       // n: source indices grouped by bucket
  int *blocksums;   // scan partials
  int nblocks;
  float *prod;      // 8n or null: per corner, weight times value of the source at each position of order
  int sms;          // multiprocessors of the device it was bound on
};

// bytes of device scratch one splat of grid d needs; products: room for the
// sources' eight contributions (32 bytes per voxel), which the sums otherwise
// form themselves
size_t splat_scratch_bytes(const Dims &d, bool products = true);
// lays out a SplatWork inside caller-provided device memory (256-aligned)
void splat_work_bind(SplatWork *w, const Dims &d, void *scratch, bool products = true);

// out = splat of img by h (three planes), background bg; stream-ordered
cudaError_t splat(const SplatWork &w, const float *img, const float *hx, const float *hy,
                  const float *hz, float *out, float bg, cudaStream_t s);
// the two halves of splat(): the bucket sort of the sources by h, kept in w,
// and the ordered per-destination sums of img, which any number of images
// splatted by the same h can share. A gather keeps the sort, but writes w's
// prod and its queue in cursor: the gathers of one w, and those of sorts that
// share a prod, are ordered on one stream.
cudaError_t splat_sort(const SplatWork &w, const float *hx, const float *hy, const float *hz,
                       cudaStream_t s);
cudaError_t splat_gather(const SplatWork &w, const float *img, const float *hx, const float *hy,
                         const float *hz, float *out, float bg, cudaStream_t s);

}  // namespace aw
