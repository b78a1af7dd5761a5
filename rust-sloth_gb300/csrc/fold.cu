// fold.cu -- one frame's draws without tiles (fold.cuh): the frame's start, the setup and
// fold of a draw, and the walk of its queued triangles.
#include "fold.cuh"
#include "launch.cuh"
#include "sloth_kernels.h"

namespace sloth {

// One block per tile: keys of tiles that are not current emptied and the tile made
// current (with all, every tile); with frame, the resets of a clear (frame_reset_kernel) too.
// Every pair of queue counters starts at zero.
__global__ void __launch_bounds__(256)
fold_begin_kernel(FrameGeom g, FrameBuffers fb, uint32_t nl_nodes, int frame, int all, uint32_t *queue_counts)
{
    const uint32_t t = blockIdx.x + pdl_begin();
    if (frame)
        for (uint32_t i = t * blockDim.x + threadIdx.x; i < nl_nodes; i += gridDim.x * blockDim.x) fb.nltree[i] = -1;
    if (t == 0 && threadIdx.x == 0) {
        for (uint32_t k = 0; k < 2 * kFoldSlots; ++k) queue_counts[k] = 0u;
        if (frame) {
            if (fb.error) *fb.error = 0u;
            *fb.fragments = 0ull;
        }
    }
    if (!all && fb.tile_gen[t] == fb.gen) return;
    block_sync();   // every thread has read the generation
    if (threadIdx.x == 0) fb.tile_gen[t] = fb.gen;
    const int tr = (int)t / g.ntx, tc = (int)t - tr * g.ntx;
    // two keys per 16-byte store: tile rows start at multiples of tw keys, tw >= 8
    const int per_row = live_keys_per_row(g.w, g.tw) / 2;
    uint4 *k0 = reinterpret_cast<uint4 *>(fb.keys + (size_t)tr * g.th * g.pitch + (size_t)tc * g.tw);
    const uint4 empty = make_uint4(~0u, ~0u, ~0u, ~0u);
    for (int i = threadIdx.x; i < g.th * per_row; i += blockDim.x) {
        const int rr = i / per_row;
        k0[(size_t)rr * (g.pitch / 2) + (i - rr * per_row)] = empty;
    }
}

// beside: the kernel before on the stream is the walk of the frame's last queue, which this
// one shares nothing with that is not a minimum, a maximum or a sum (its own queue and
// counters, its own records; the mesh is written by nobody), so it runs beside it, and waits
// for it only before it ends: whoever waits for this kernel has waited for all before it.
// Both are bound by latency, with most of the GPU idle: 16 models at 1280x720 252 -> 205 us.
template <int kWarps>
__global__ void __launch_bounds__(32 * kWarps)
fold_setup_kernel(MeshDev mesh, Mat4 M, uint32_t tri_base, FrameGeom g, FrameBuffers fb, FoldQueue queue, int beside)
{
    uint32_t zero = 0u;
    if (beside) pdl_trigger();
    else zero = pdl_begin();
    fold_triangles<kWarps>(mesh, M, blockIdx.x * kFoldTris + zero, tri_base, g, fb, queue, 0u);
    if (beside) pdl_wait();
}

// The queued triangles' items over the warps of the grid, the large ones' first.  next: the
// counters of the draw before, emptied here for the draw after the next (the next one's setup
// may run already).
struct FoldFrame {
    FrameGeom g;
    FrameBuffers fb;
};

// 2^22 warps' worth of items above those of the most triangles a draw folds
static_assert((uint64_t)kFoldMaxTrianglesMade * kFoldParts + (32ull << 22) < (1ull << 32) &&
                  kFoldMaxTrianglesMade >= kFoldMaxTriangles && kFoldParts >= kFoldMidParts,
              "32-bit items");

__global__ void __launch_bounds__(256)
fold_large_kernel(const __grid_constant__ FoldFrame f, FoldQueue queue, uint32_t *next)
{
    const uint32_t first = (blockIdx.x * blockDim.x + threadIdx.x + pdl_begin()) >> 5;
    if (blockIdx.x == 0 && threadIdx.x < 2) next[threadIdx.x] = 0u;
    const uint32_t frags = fold_queue_walk<uint32_t>(queue, first, (gridDim.x * blockDim.x) >> 5,
                                           [&](uint32_t) -> const FoldFrame & { return f; });
    add_frags_warp(frags, f.fb.fragments);
}

// The queue of a frame's draw number `draw`: half of the cap entries and one pair of counters.
static FoldQueue fold_queue(uint32_t *queue, uint32_t cap, uint32_t *queue_counts, uint32_t draw)
{
    const uint32_t half = cap / 2;
    return FoldQueue{queue + (draw & 1u) * half, nullptr, queue_counts + 2 * (draw % kFoldSlots), half};
}

cudaError_t launch_fold_begin(const FrameGeom &g, const FrameBuffers &fb, bool frame, bool all,
                              uint32_t *queue_counts, cudaStream_t s)
{
    return launch_pdl(fold_begin_kernel, dim3((unsigned)(g.ntx * g.nty)), dim3(256), 0, s, g, fb,
                      2u * (uint32_t)g.nl_size, frame ? 1 : 0, all ? 1 : 0, queue_counts);
}

cudaError_t launch_fold_setup(const MeshDev &mesh, const Mat4 &M, uint32_t tri_base, const FrameGeom &g,
                              const FrameBuffers &fb, uint32_t *queue, uint32_t cap, uint32_t *queue_counts,
                              uint32_t draw, bool beside, cudaStream_t s)
{
    if (mesh.ntri == 0) return cudaSuccess;
    const FoldQueue q = fold_queue(queue, cap, queue_counts, draw);
    const uint32_t blocks = (mesh.ntri + kFoldTris - 1) / kFoldTris;
    return launch_pdl(fold_setup_kernel<4>, dim3(blocks), dim3(128), kFoldSmemBytes, s, mesh, M, tri_base, g, fb, q,
                      beside ? 1 : 0);
}

cudaError_t launch_fold_large(const FrameGeom &g, const FrameBuffers &fb, uint32_t *queue, uint32_t cap,
                              uint32_t *queue_counts, uint32_t draw, cudaStream_t s)
{
    const FoldQueue q = fold_queue(queue, cap, queue_counts, draw);
    return launch_pdl(fold_large_kernel, dim3(4u * (unsigned)device_sm_count()), dim3(256), 0, s, FoldFrame{g, fb}, q,
                      queue_counts + 2 * ((draw + kFoldSlots - 1) % kFoldSlots));
}

}  // namespace sloth
