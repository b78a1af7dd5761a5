// noalloc.cu -- sloth_render_noalloc: one frame of one triangle soup with no device
// allocation.
//
// Some callers cannot let a library call cudaMalloc:
//  - hosts that give the renderer a fixed memory budget at start-up and forbid
//    allocation afterwards (plug-ins, embedded viewers);
//  - frame loops that cannot afford the device-wide synchronisation cudaMalloc/cudaFree
//    imply;
//  - programs whose device memory is fully reserved by a framework's caching pool.
// For them this entry point takes device inputs and outputs from the caller and keeps
// every intermediate buffer in one file-scope __device__ array of a fixed size
// (kScratchBytes).  That array exists on every GPU that loads the library, until the
// process exits.  It has no counterpart in the reference.
//
// Scratch layout (byte offsets into g_noalloc_scratch):
//   records   kMaxTri x 96 B          per-triangle setup records
//   (free)    kMaxTri x 4 B           unused, as are the tile counts below: the header states
//                                     the array's size
//   keys      kMaxCells x 8 B         depth keys (tiles padded to 64x32 cells)
//   queue     kMaxTri x 4 B + 24 B    triangles too large for their block, and their counters
//   tile_gen  kMaxTiles x 4 B         tile generations (cleared every call)
//   nltree    2*kMaxNl x 4 B          newline segment tree (cleared every call)
//   frags     8 B                     fragment counter (cleared every call)
#include "sloth_gpu.h"
#include "sloth_internal.cuh"
#include "sloth_kernels.h"

namespace sloth {
namespace {

constexpr uint32_t kMaxTri = SLOTH_NOALLOC_MAX_TRIANGLES;
constexpr uint32_t kMaxCells = SLOTH_NOALLOC_MAX_DEPTH_CELLS;
constexpr uint32_t kMaxNl = SLOTH_NOALLOC_MAX_HEIGHT;            // power of two
constexpr uint32_t kMaxTiles = kMaxCells / (kTileW * kTileH);

constexpr size_t align256(size_t n) { return (n + 255) & ~size_t(255); }
constexpr size_t kOffRecords = 0;
constexpr size_t kOffRows = align256(kOffRecords + (size_t)kMaxTri * sizeof(TriRecord));
constexpr size_t kOffKeys = align256(kOffRows + (size_t)kMaxTri * 4);
constexpr size_t kOffCount = align256(kOffKeys + (size_t)kMaxCells * sizeof(uint64_t));
constexpr size_t kOffOffset = align256(kOffCount + (size_t)kMaxTiles * 4);
constexpr size_t kOffCursor = align256(kOffOffset + ((size_t)kMaxTiles + 1) * 4);
constexpr size_t kOffQueue = align256(kOffCursor + (size_t)kMaxTiles * 4);
constexpr size_t kOffQCount = align256(kOffQueue + (size_t)kMaxTri * 4);
constexpr size_t kOffGen = align256(kOffQCount + 2 * kFoldSlots * 4);
constexpr size_t kOffNl = align256(kOffGen + (size_t)kMaxTiles * 4);
constexpr size_t kOffFrags = align256(kOffNl + 2 * (size_t)kMaxNl * 4);
constexpr size_t kScratchBytes = align256(kOffFrags + 8);
static_assert(kScratchBytes == SLOTH_NOALLOC_SCRATCH_BYTES, "header states the scratch size");

}  // namespace

// The scratch every call uses.  In host code this name is only a stand-in for the
// device symbol; its device address comes from cudaGetSymbolAddress (scratch_on()), with
// the device the caller made current.
static __device__ __align__(256) unsigned char g_noalloc_scratch[kScratchBytes];

namespace {

// Device address of g_noalloc_scratch for the current device, looked up on every call with
// the caller's device current.  cudaGetSymbolAddress allocates nothing; an address kept
// from an earlier call could belong to a context that cudaDeviceReset (or a driver-API
// caller switching contexts) has since replaced, and kernels given it would fault.
cudaError_t scratch_on(unsigned char **out)
{
    void *p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess) return e;
    *out = static_cast<unsigned char *>(p);
    return cudaSuccess;
}

}  // namespace
}  // namespace sloth

using namespace sloth;

extern "C" sloth_status sloth_render_noalloc(const float *x, const float *y, const float *z,
                                             uint32_t ntri, const uint8_t *rgb, const float m[16],
                                             uint32_t width, uint32_t height, int image,
                                             uint32_t *cells, float *zbuf, int32_t *winner, void *stream)
{
    if (!m || !cells || !zbuf || !winner || (ntri && (!x || !y || !z || !rgb)))
        return SLOTH_ERR_INVALID_ARGUMENT;
    if (width < 1 || height < 1 || width > SLOTH_MAX_DIM || height > SLOTH_NOALLOC_MAX_HEIGHT)
        return SLOTH_ERR_LIMIT;
    if (ntri > kMaxTri) return SLOTH_ERR_LIMIT;
    FrameGeom g{};
    g.w = (int32_t)width;
    g.h = (int32_t)height;
    g.image = image ? 1 : 0;
    g.tw = kTileW;
    g.th = kTileH;
    g.ntx = (g.w + g.tw - 1) / g.tw;
    g.nty = (g.h + g.th - 1) / g.th;
    g.pitch = g.ntx * g.tw;
    g.nl_size = 1;
    while (g.nl_size < g.h) g.nl_size <<= 1;
    const uint64_t padded = (uint64_t)g.pitch * g.nty * g.th;
    if (padded > kMaxCells) return SLOTH_ERR_LIMIT;

    unsigned char *base = nullptr;
    if (scratch_on(&base) != cudaSuccess) return SLOTH_ERR_CUDA;
    cudaStream_t s = static_cast<cudaStream_t>(stream);

    FrameBuffers fb{};
    fb.records = reinterpret_cast<TriRecord *>(base + kOffRecords);
    fb.keys = reinterpret_cast<uint64_t *>(base + kOffKeys);
    fb.tile_gen = reinterpret_cast<uint32_t *>(base + kOffGen);
    fb.nltree = reinterpret_cast<int32_t *>(base + kOffNl);
    fb.fragments = reinterpret_cast<unsigned long long *>(base + kOffFrags);
    fb.z_out = zbuf;
    fb.cells_out = cells;
    fb.winner_out = winner;
    fb.gen = 1;
    // The array keeps the previous call's contents: every tile's keys and the frame's
    // counters are reset first.  The draw goes without tiles (fold.cuh): a raster of one CTA
    // per tile over the whole soup took 1323 us for 20,000 triangles at 640x360, all of it
    // record loads of triangles that miss the tile; this takes 21 us.
    uint32_t *queue = reinterpret_cast<uint32_t *>(base + kOffQueue);
    uint32_t *queue_counts = reinterpret_cast<uint32_t *>(base + kOffQCount);
    if (launch_fold_begin(g, fb, true, true, queue_counts, s) != cudaSuccess) return SLOTH_ERR_CUDA;
    Mat4 M;
    for (int i = 0; i < 16; ++i) M.m[i] = m[i];
    const MeshDev md{x, y, z, nullptr, rgb, 3 * ntri, ntri};
    if (ntri && (launch_fold_setup(md, M, 0, g, fb, queue, 2 * kMaxTri, queue_counts, 0, false, s) != cudaSuccess ||
                 launch_fold_large(g, fb, queue, 2 * kMaxTri, queue_counts, 0, s) != cudaSuccess))
        return SLOTH_ERR_CUDA;
    if (launch_resolve(g, fb, s) != cudaSuccess) return SLOTH_ERR_CUDA;
    return SLOTH_OK;
}
