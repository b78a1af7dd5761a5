// newline.cuh -- newline sentinels (src/rasterizer.rs:89-91), shared by the single-frame and
// batched kernels.  In image mode every row y in [y0,y1) of every triangle gets frame cell
// y*w+1 = '\n' after the row's samples.  The resolve needs, per row, the last triangle in
// draw order that wrote it: the maximum draw index whose [y0,y1) contains y.  Each triangle
// folds its interval into a max segment tree with O(log h) node updates (canonical
// decomposition); a row's value is the maximum over its leaf-to-root path.
#pragma once

#include "record.cuh"

namespace sloth {

// Triangles per block of the newline kernel.  A block builds a tree of its chunk in shared memory (2n nodes) and
// merges the nodes it touched into the frame's tree.
constexpr uint32_t kNewlineChunk = 8192;
// The same for a newline part of a fill or fold, whose blocks have a quarter of the threads:
// the part must not outlast the rest of its launch, and in blocks of 8192 it did (us a frame of
// a soup, 8192 / 2048 / 1024 / 512 a block: 8k triangles at 3840x1426 152 / 112 / 107 / 102,
// 96k there 204 / 163 / 156 / 153, 96k at 1280x720 148 / 118 / 112 / 112).
constexpr uint32_t kNewlineFillChunk = 1024;
// The largest tree, in bytes, that a fill or fold kernel takes into its own blocks as one of
// its parts: every block of the launch holds that much shared memory, and at 32 KB (frames
// of up to 4096 rows) six still fit an SM.  Taller frames launch the newline kernel, and so
// do more triangles than kNewlinePartTriangles: beside the rest on a stream of its own it
// fills the raster's gaps too (a million triangles: 17 us as a part of the fill, none
// there), which for fewer is not worth the fork and the join.
constexpr size_t kNewlinePartBytes = 32 * 1024;
constexpr uint32_t kNewlinePartTriangles = 1u << 17;
// The largest tree the newline kernel holds in shared memory; above it the frame's tree is
// updated directly.
constexpr size_t kNewlineSharedBytes = 128 * 1024;

inline size_t newline_tree_bytes(int nl_size) { return 2 * (size_t)nl_size * sizeof(int32_t); }

// Positions [lo, hi) of setup's order of a mesh: rows holds each position's packed sample
// rows (4 bytes a triangle, setup wrote them), order maps a position to its triangle (null:
// the same), base is the draw index of the mesh's first triangle.
template <bool kShared>
__device__ __forceinline__ void newline_block(int32_t *stree, int n, uint32_t lo, uint32_t hi,
                                              const uint32_t *__restrict__ order, const uint32_t *__restrict__ rows,
                                              uint32_t base, int32_t *tree)
{
    int32_t *t = kShared ? stree : tree;
    if (kShared) {
        for (int i = threadIdx.x; i < 2 * n; i += blockDim.x) stree[i] = -1;
        block_sync();
    }
    for (uint32_t p = lo + threadIdx.x; p < hi; p += blockDim.x) {
        const int32_t v = (int32_t)(base + (order ? __ldg(order + p) : p));
        const uint32_t yr = __ldg(rows + p);
        nltree_update(t, n, (int)(yr & 0xffffu), (int)(yr >> 16), v, kShared);
    }
    if (kShared) {
        block_sync();
        for (int i = threadIdx.x; i < 2 * n; i += blockDim.x) {
            const int32_t v = stree[i];
            if (v >= 0 && *(volatile int32_t *)&tree[i] < v) atomicMax(&tree[i], v);
        }
    }
}

}  // namespace sloth
