// Device side of a batched launch shared by batch.cu and the line-specialised batched
// kernels: the header of a launch's instances and the walk over their descriptors.
#pragma once

#include "opo_internal.h"

namespace opo {

// One launch's share of a descriptor array: instances [first, first + ninst) with their
// tile prefix at prefix[pfirst ...] (starting at 0), total_tiles tiles.
struct BatchHeader {
    unsigned ninst;
    unsigned total_tiles;
    unsigned first;
    unsigned pfirst;
};

template <typename Args> __host__ __device__ constexpr unsigned desc_bytes() { return (unsigned)((sizeof(Args) + 127) / 128 * 128); }

template <typename Args> __device__ __forceinline__ void stage_desc(const Args *src, Args *dst)
{
    const unsigned *s = reinterpret_cast<const unsigned *>(src);
    unsigned *d = reinterpret_cast<unsigned *>(dst);
    for (unsigned k = threadIdx.x; k < sizeof(Args) / 4; k += blockDim.x) d[k] = s[k];
}

// Largest i < ninst with prefix[i] <= gt.
__device__ __forceinline__ int find_inst(const unsigned *prefix, unsigned ninst, unsigned gt)
{
    int lo = 0, hi = (int)ninst - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (__ldg(prefix + mid) <= gt) lo = mid;
        else hi = mid - 1;
    }
    return lo;
}

// The instance of the ascending tile numbers a persistent CTA walks: its tiles [begin, end)
// are kept, so a tile of the same instance costs one comparison.
struct InstWalk {
    int cur = -1;
    unsigned begin = 0, end = 0;
    // Moves to the instance of tile gt; true when it is another one.
    __device__ __forceinline__ bool seek(const unsigned *prefix, unsigned ninst, unsigned gt)
    {
        if (gt < end) return false;
        cur = find_inst(prefix, ninst, gt);
        begin = __ldg(prefix + cur);
        end = __ldg(prefix + cur + 1);
        return true;
    }
};

}  // namespace opo
