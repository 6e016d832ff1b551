// be_uf2d.cu -- 2D Block-Equivalence labeling, union-find form (8-connectivity, 2x2 blocks).
// The pipeline itself is in be_uf2d_impl.cuh, instantiated here for three tile shapes
// (32 x 128, 64 x 64 and 16 x 256 blocks) that the autotuner chooses between, and once on pixels for
// 4-connectivity (the pixel label-equivalence and run-equivalence forms).
//
// Replaces the reference's LBEQ2_Init / LBEQ2_Scan / LBEQ2_Analyze / LBEQ2_SetFinalLabels
// (LabelingAlgs.cl:176-319) and their host loop (LabelingAlgs.cpp:989-1084) with four launches:
//
//   k_tile_local_2d   one CTA per 64x256-pixel tile: 16-byte loads, 2x2 block masks, runs of blocks
//                     and their links by bit operations; runs numbered in the order of their first
//                     pixels; each run's first link becomes its parent by a plain store (a forest),
//                     the other links are unions in shared memory (smaller number wins); writes
//                     the tile's bit words, the root run of every run, a bitmap of the root runs and
//                     the root count per segment, and exports border components as nodes.
//   k_merge_2d        unions nodes across tile borders (global union-find after Rem's
//                     algorithm, smaller key wins); every root that gets linked leaves its segment
//                     count and its root bitmap.
//   k_scan_flatten_2d single-pass exclusive scan of the segment counts (be_scan.cuh) and, in
//                     the same launch, every linked node pointed at its global root (pointer
//                     jumping).
//   k_tile_write_2d   one CTA per tile: the label of every run, then the int32 labels with 16-byte
//                     stores.
//
// Canonical numbering.  A component's label is 1 + the number of components whose first pixel in
// raster order precedes its own.  Within a segment -- the part of a pixel row in one tile -- runs are
// numbered in the order of their first pixels, and a component's root is the run of its first
// pixel, so the label is the exclusive prefix of the segments' root counts plus the rank of the root's
// bit among the segment's bits: no pixel positions are stored or sorted.
#include "be_common.cuh"
#include "be_kernels.h"
#include "be_scan.cuh"

#include "be_api_internal.h"

#include <algorithm>

namespace be {

namespace s32x128 {
constexpr int CELL = 2, TBW = 128, TBH = 32;
#include "be_uf2d_impl.cuh"
}  // namespace s32x128

namespace s64x64 {
constexpr int CELL = 2, TBW = 64, TBH = 64;
#include "be_uf2d_impl.cuh"
}  // namespace s64x64

namespace s16x256 {
constexpr int CELL = 2, TBW = 256, TBH = 16;
#include "be_uf2d_impl.cuh"
}  // namespace s16x256

// 4-connectivity: pixel cells, 64 x 128 pixels, one thread per 32 pixels (256 threads).
namespace p64x128 {
constexpr int CELL = 1, TBW = 128, TBH = 64;
#include "be_uf2d_impl.cuh"
}  // namespace p64x128

const Shape2D kShapes2D[kNumShapes2D + 1] = {{256, 64}, {128, 128}, {512, 32}, {128, 64}};

Geometry uf2d_geometry(int shape)
{
    switch (shape) {
    case 1: return s64x64::geometry();
    case 2: return s16x256::geometry();
    case kShapePixel2D: return p64x128::geometry();
    default: return s32x128::geometry();
    }
}

cudaError_t uf2d_launch(int shape, const ImgList2D &L, const Work &w, int sms, bool persistent,
                        cudaStream_t s, cudaEvent_t *ev)
{
    switch (shape) {
    case 1: return s64x64::launch(L, w, sms, persistent, s, ev);
    case 2: return s16x256::launch(L, w, sms, persistent, s, ev);
    case kShapePixel2D: return p64x128::launch(L, w, sms, persistent, s, ev);
    default: return s32x128::launch(L, w, sms, persistent, s, ev);
    }
}

}  // namespace be
