// fold.cu -- one frame's draws without tiles (fold.cuh): the frame's start, the setup and
// fold of a draw, and the walk of its queued triangles.
#include "fold.cuh"
#include "launch.cuh"
#include "sloth_kernels.h"

namespace sloth {

// One block per tile: keys of tiles that are not current emptied and the tile made
// current (with all, every tile); with frame, the resets of a clear (frame_reset_kernel) too.  The queue counters
// of both parities start at zero.
__global__ void __launch_bounds__(256)
fold_begin_kernel(FrameGeom g, FrameBuffers fb, uint32_t nl_nodes, int frame, int all, uint32_t *queue_counts)
{
    const uint32_t t = blockIdx.x + pdl_begin();
    if (frame)
        for (uint32_t i = t * blockDim.x + threadIdx.x; i < nl_nodes; i += gridDim.x * blockDim.x) fb.nltree[i] = -1;
    if (t == 0 && threadIdx.x == 0) {
        queue_counts[0] = queue_counts[1] = queue_counts[2] = queue_counts[3] = 0u;
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

template <int kWarps>
__global__ void __launch_bounds__(32 * kWarps)
fold_setup_kernel(MeshDev mesh, Mat4 M, uint32_t tri_base, FrameGeom g, FrameBuffers fb, FoldQueue queue)
{
    fold_triangles<kWarps>(mesh, M, blockIdx.x * kFoldTris + pdl_begin(), tri_base, g, fb, queue, 0u);
}

// The queued triangles' items over the warps of the grid, the large ones' first.  next: the
// counters the frame's next draw queues with, emptied here (the draw after that reuses
// this one's).
struct FoldFrame {
    FrameGeom g;
    FrameBuffers fb;
};

__global__ void __launch_bounds__(256)
fold_large_kernel(const __grid_constant__ FoldFrame f, FoldQueue queue, uint32_t *next)
{
    const uint32_t first = (blockIdx.x * blockDim.x + threadIdx.x + pdl_begin()) >> 5;
    if (blockIdx.x == 0 && threadIdx.x < 2) next[threadIdx.x] = 0u;
    const uint32_t frags = fold_queue_walk(queue, first, (gridDim.x * blockDim.x) >> 5,
                                           [&](uint32_t) -> const FoldFrame & { return f; });
    add_frags_warp(frags, f.fb.fragments);
}

cudaError_t launch_fold_begin(const FrameGeom &g, const FrameBuffers &fb, bool frame, bool all,
                              uint32_t *queue_counts, cudaStream_t s)
{
    return launch_pdl(fold_begin_kernel, dim3((unsigned)(g.ntx * g.nty)), dim3(256), 0, s, g, fb,
                      2u * (uint32_t)g.nl_size, frame ? 1 : 0, all ? 1 : 0, queue_counts);
}

cudaError_t launch_fold_setup(const MeshDev &mesh, const Mat4 &M, uint32_t tri_base, const FrameGeom &g,
                              const FrameBuffers &fb, uint32_t *queue, uint32_t cap, uint32_t *queue_counts,
                              int parity, cudaStream_t s)
{
    if (mesh.ntri == 0) return cudaSuccess;
    const FoldQueue q{queue, nullptr, queue_counts + 2 * parity, cap};
    const uint32_t blocks = (mesh.ntri + kFoldTris - 1) / kFoldTris;
    return launch_pdl(fold_setup_kernel<4>, dim3(blocks), dim3(128), kFoldSmemBytes, s, mesh, M, tri_base, g, fb, q);
}

cudaError_t launch_fold_large(const FrameGeom &g, const FrameBuffers &fb, uint32_t *queue, uint32_t cap,
                              uint32_t *queue_counts, int parity, cudaStream_t s)
{
    const FoldQueue q{queue, nullptr, queue_counts + 2 * parity, cap};
    return launch_pdl(fold_large_kernel, dim3(4u * (unsigned)device_sm_count()), dim3(256), 0, s, FoldFrame{g, fb}, q,
                      queue_counts + 2 * (parity ^ 1));
}

}  // namespace sloth
