// resolve.cu -- depth keys -> depth buffer, frame cells and winners (one frame).
// The per-cell rule is in resolve_common.cuh.
#include <algorithm>

#include "launch.cuh"
#include "resolve_common.cuh"

namespace sloth {

// Runs of kRun frame cells; each warp takes 32 consecutive runs (resolve_run).  An
// even-width frame goes by pairs of cells instead, kEvenPairs per thread (resolve_even).
// The winner's key and record are two dependent loads from L2 or memory, so what counts is
// the warps that wait on them at once: eight blocks an SM with one pair a thread (32
// registers) take 34 us for 3840x2160 over a million triangles, four blocks with four pairs
// 47; an odd 1921x1079 takes 18 at eight blocks, 24 at four.
constexpr int kRun = 2;
constexpr int kEvenPairs = 1;

template <bool kEven>
__global__ void __launch_bounds__(256, 8) resolve_kernel(FrameGeom g, FrameBuffers fb, int vec)
{
    const uint32_t tid = threadIdx.x + pdl_begin(), ncells = frame_cells(g);
    if (kEven) {
        const uint32_t npairs = ncells / 2 + (ncells & 1u), span = blockDim.x * kEvenPairs;
        for (uint64_t base = (uint64_t)blockIdx.x * span; base < npairs; base += (uint64_t)gridDim.x * span)
            resolve_even<kEvenPairs, true>(g, fb, (uint32_t)base + tid, blockDim.x, npairs, vec != 0);
        return;
    }
    const uint32_t nruns = ncells / kRun + (ncells % kRun != 0);
    const int lane = threadIdx.x & 31;
    for (uint64_t base = (uint64_t)blockIdx.x * blockDim.x; base < nruns; base += (uint64_t)gridDim.x * blockDim.x) {
        const uint32_t p = (uint32_t)base + tid;
        resolve_run<kRun, true>(g, fb, p, p < nruns, lane, vec != 0);
    }
}

cudaError_t launch_resolve(const FrameGeom &g, const FrameBuffers &fb, cudaStream_t s)
{
    const uint64_t ncells = (uint64_t)g.w * g.h + (g.image ? g.h : 0);
    if (ncells == 0) return cudaSuccess;
    const uint64_t per_block = 256ull * kRun * ((g.w & 1) ? 1 : kEvenPairs);   // cells
    uint64_t blocks = (ncells + per_block - 1) / per_block;
    const uint64_t cap = 64ull * (uint64_t)device_sm_count();   // eight resident CTAs per SM, eight waves
    if (blocks > cap) blocks = cap;
    const int vec = ((reinterpret_cast<uintptr_t>(fb.cells_out) | reinterpret_cast<uintptr_t>(fb.z_out) |
                      reinterpret_cast<uintptr_t>(fb.winner_out)) & (4u * kRun - 1u)) == 0;
    return launch_pdl((g.w & 1) ? resolve_kernel<false> : resolve_kernel<true>, dim3((unsigned)blocks), dim3(256), 0, s, g,
                      fb, vec);
}

// A small frame's buffers and the error word into one page-locked buffer, by words of 16
// bytes (the sources start allocations, the parts of the destination 16-byte lines; a part's
// last line is copied by words).  Three or four copies of a few kilobytes cost the host and
// the copy engine about 10 us each; this is one launch behind the resolve.
__global__ void __launch_bounds__(256) readback_kernel(ReadBack r)
{
    const uint32_t i0 = blockIdx.x * blockDim.x + threadIdx.x + pdl_begin(), step = gridDim.x * blockDim.x;
    if (i0 == 0) *r.error_out = *r.error;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        if (!r.n[k]) continue;
        const uint32_t n = r.n[k];
        for (uint32_t i = i0; i < n / 4; i += step)
            reinterpret_cast<uint4 *>(r.out[k])[i] = reinterpret_cast<const uint4 *>(r.in[k])[i];
        if (i0 < (n & 3u)) r.out[k][(n & ~3u) + i0] = r.in[k][(n & ~3u) + i0];
    }
}

cudaError_t launch_readback(const ReadBack &r, cudaStream_t s)
{
    const uint32_t most = (std::max(r.n[0], std::max(r.n[1], r.n[2])) + 3) / 4;
    const uint32_t blocks = std::max(1u, std::min((most + 255) / 256, (uint32_t)device_sm_count()));
    return launch_pdl(readback_kernel, dim3(blocks), dim3(256), 0, s, r);
}

}  // namespace sloth
