// fold_items.h -- how the work items of queued triangles are numbered, for the walk of a
// fold's queue (fold.cuh) and the overflow folds of the tile rasters (raster.cu, batch.cu).
//
// The frames of a batch share one queue, and from 8,388,608 large triangles on kFoldParts items
// each are 2^32 or more: their numbers are 64-bit.  One draw's fold stops at 2^20 triangles,
// and 32 bits do: its walks, one after another, are timed by their length (with 64 the sixteen
// of 16 models at 1280x720 took 7 us of 160 more; a batch has one, and 59 views of 151x81 take
// 94 us either way).
// Plain C++, so that the numbering is tested on the host at sizes no test draws.
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define SLOTH_HD __host__ __device__ __forceinline__
#else
#define SLOTH_HD inline
#endif

namespace sloth {

// Items of a large queued triangle, and of one of the others (fold.cuh says why these).
constexpr uint32_t kFoldParts = 512, kFoldMidParts = 8;
// Items of a large triangle of an overflow fold.
constexpr uint32_t kOverflowParts = 64;

// n / d; the 64-bit division, many times as long, only for the counts that need it.
SLOTH_HD uint32_t item_part(uint32_t n, uint32_t d) { return n / d; }
SLOTH_HD uint32_t item_part(uint64_t n, uint32_t d)
{
    return n >> 32 ? (uint32_t)(n / d) : (uint32_t)n / d;
}

// The items of a fold's queue: every part of the large triangles, part after part, then of
// the others (one item each when `whole`).  The large ones are queued from the front of the
// cap entries, the others from the back.  Index: a type that all + 32 items a warp of the
// walk's grid fits in.
template <class Index>
struct FoldItems {
    uint32_t large, mid, cap;
    Index cut, all;   // the large ones' items, all items

    SLOTH_HD FoldItems(uint32_t large_, uint32_t mid_, uint32_t cap_, bool whole)
        : large(large_), mid(mid_), cap(cap_), cut((Index)large_ * kFoldParts),
          all(cut + (Index)mid_ * (whole ? 1u : kFoldMidParts))
    {
    }
    // Queue entry and part of item it (below all).
    SLOTH_HD uint32_t entry(Index it, uint32_t &part) const
    {
        if (it < cut) {
            part = item_part(it, large);
            return (uint32_t)it - part * large;
        }
        it -= cut;
        part = item_part(it, mid);
        return cap - 1u - ((uint32_t)it - part * mid);
    }
};

// The items of the large queue of a draw that outgrew its entry buffer: kOverflowParts of
// each triangle, those queued from the front first.
struct OverflowItems {
    uint32_t front, cap;
    uint64_t all;

    SLOTH_HD OverflowItems(uint32_t front_, uint32_t back, uint32_t cap_)
        : front(front_), cap(cap_), all((uint64_t)(front_ + back) * kOverflowParts)
    {
    }
    SLOTH_HD uint32_t entry(uint64_t it, uint32_t &part) const
    {
        const uint32_t k = (uint32_t)(it / kOverflowParts);
        part = (uint32_t)it % kOverflowParts;
        return k < front ? k : cap - 1u - (k - front);
    }
};

}  // namespace sloth
