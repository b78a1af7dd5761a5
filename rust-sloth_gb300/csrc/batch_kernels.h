// batch_kernels.h -- device tables and launchers of the batched (many frames) path.
//
// A batch is a list of frames (viewport, image mode, utransform) and, per frame, an
// ordered list of draws (mesh, transform) -- the reference's per-frame loop over its
// mesh queue (src/main.rs:76-83) for many frames or views at once.  Every frame keeps its
// own depth keys, newline tree, records and outputs; draw indices inside a frame are
// frame-local, so every frame is bit-identical to drawing it alone.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "sloth_kernels.h"

namespace sloth {

struct BatchFrame {
    FrameGeom g;
    FrameBuffers fb;           // pointers into the batch's buffers, records offset to the frame
    uint32_t tile_off;         // first global tile of the frame
    uint32_t rec_off;          // first global record of the frame
    uint32_t first_draw;       // the frame's first draw
    uint32_t ndraws;
    uint64_t z_off;            // first depth cell of the frame in the batch's depth-cell order
    int32_t vec;               // the frame's outputs start on 8-byte boundaries: the resolve
                               // writes 2 cells per store
};

struct BatchDraw {
    MeshDev mesh;
    uint32_t frame;
    uint32_t rec_off;          // global record of the draw's first triangle
    uint32_t local_base;       // frame-local draw index of the draw's first triangle
};

struct BatchDev {
    const BatchFrame *frames;
    const BatchDraw *draws;
    const Mat4 *mats;          // per draw: utransform * transform
    uint32_t nframes, ndraws;
    uint32_t total_tiles;
    const uint32_t *frame_tile_off;   // nframes + 1 (for tile -> frame lookups)
    BinBuffers bb;             // global tile arrays and entries
    uint32_t *large_frame;     // frame of each large-queue entry
    volatile uint32_t *status; // pinned host words: [0] a render's entries outgrew their capacity,
                               // [1] a raster block gave up waiting for its keys
    uint32_t *queue;           // the persistent raster's next item (zeroed by the fill)
    uint32_t *fill_count;      // entries of bb.fill_list (zeroed at the start of a render)
    int depth_cull;
    int tpb;                   // triangles per setup block (the triangle block table's step)
    int direct_max;            // the frames' FrameGeom::direct_max (the same for every frame)
    uint32_t resolve_chunk;    // cells per resolve block (the resolve table's step)
    uint32_t newline_chunk;    // triangles per newline block (the newline table's step)
};

// What a render empties before it starts, in one launch.
struct BatchReset {
    uint32_t *tile_count, *tile_cursor, *tile_gen;
    uint32_t ntiles, gen;      // the generation every tile gets
    int32_t *nltree;
    uint32_t nnl;
    uint32_t *large_count, *fill_count;
    unsigned long long *fragments;
    float4 *mats;              // device matrices, and the pinned ones they are copied from
    const float4 *mats_host;
    uint32_t nmats;            // in float4
    uint4 *keys;               // keys to empty: n4 16-byte stores, in the even half of each
    uint64_t n4;               // tile row (2^half_shift stores) or, half_shift 63, all in a row
    uint32_t half_shift;
};
cudaError_t launch_batch_reset(const BatchReset &r, cudaStream_t s);

// Block tables: one int2 (item, start) per block, built on the host.
cudaError_t launch_batch_setup(const BatchDev &b, const int2 *blocks, uint32_t nblocks, cudaStream_t s);
// whether the fill's and the fold's blocks take the newline table (by kBatchNewlineFillChunk)
// of ntri triangles and trees of max_nl leaves; launch_batch_newline when they do not
bool batch_newline_part(uint64_t ntri, int max_nl);
cudaError_t launch_batch_newline(const BatchDev &b, const int2 *blocks, uint32_t nblocks, int max_nl,
                                 cudaStream_t s);
cudaError_t launch_batch_count_large(const BatchDev &b, cudaStream_t s);
// the tile entries, the raster items and nnewline blocks of the newline table (0 unless
// batch_newline_part)
cudaError_t launch_batch_fill(const BatchDev &b, const int2 *newline, uint32_t nnewline, int max_nl, cudaStream_t s);
cudaError_t launch_batch_raster(const BatchDev &b, int tw, int th, bool persistent, cudaStream_t s);
// frames without tiles: setup and fold (by blocks of `warps` warps, 4 or 1, over a
// kFoldBlockTris table; 0: by the setup kernel over the setup table), which queues the larger
// triangles in bb.large_queue and large_frame, then those
cudaError_t launch_batch_fold_setup(const BatchDev &b, const int2 *blocks, uint32_t nblocks, int warps,
                                    cudaStream_t s);
cudaError_t launch_batch_fold_large(const BatchDev &b, const int2 *newline, uint32_t nnewline, int max_nl,
                                    cudaStream_t s);
// odd: some frame has an odd width
cudaError_t launch_batch_resolve(const BatchDev &b, const int2 *blocks, uint32_t nblocks, bool odd, cudaStream_t s);
cudaError_t prepare_batch_kernels();

constexpr uint32_t kBatchNewlineChunk = 8192;   // triangles per newline block (kNewlineChunk)
constexpr uint32_t kBatchNewlineFillChunk = 1024;   // the same as a part of the fill (kNewlineFillChunk)
constexpr uint32_t kBatchResolveChunk = 8192;   // cells per resolve block (four rounds of its threads)
constexpr uint32_t kBatchResolveSmall = 2048;   // the same (one round) for batches of few blocks
constexpr uint32_t kFoldBlockTris = 32;         // triangles per block of a small fold's table
// Triangles of a batch up to which it has that table, up to which its blocks may be of four
// warps, and from which they may be of one (batch_folds)
constexpr uint32_t kFoldTableTriangles = 1u << 20;
constexpr uint32_t kFoldMany4 = 1u << 18;
constexpr uint32_t kFoldMany = 1u << 16;

}  // namespace sloth
