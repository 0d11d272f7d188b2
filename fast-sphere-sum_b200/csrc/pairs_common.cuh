// pairs_common.cuh -- what the two pair engines share: packing of a work
// item's source segments into tiles, and their kernels' launch.
#pragma once
#include <cuda_runtime.h>

#include "device_common.cuh"
#include "kernels.h"

namespace fss {

// Packing of a work item's sources into tiles, by one warp.  A window of 32 segments is held one per lane as the range [lo,
// hi) of its sources not yet packed (kind 0 resolved through leaf_start); the
// window after it is loaded in advance, so that a tile's packing does not
// wait for memory.  A warp scan places the window's ranges back to back and
// each lane issues the bulk copy of its piece; the segment cut by the end of
// the tile keeps its rest.
struct Window {
    int lo, hi, nlo, nhi;  // this lane's segment, and the one 32 further on
    int g;                 // first segment not in either window
};
__device__ __forceinline__ void window_load(const Segment* __restrict__ segs, const int32_t* __restrict__ leaf_start,
                                            int g1, Window& w) {
    w.lo = w.nlo;
    w.hi = w.nhi;
    const int gi = w.g + int(threadIdx.x & 31);
    w.nlo = w.nhi = 0;
    if (gi < g1) {
        const Segment sg = segs[gi];
        w.nlo = sg.kind == 0 ? leaf_start[sg.a] : sg.a;
        w.nhi = sg.kind == 0 ? leaf_start[sg.b] : sg.b;
    }
    w.g = min(w.g + 32, g1 + 32);
}
__device__ __forceinline__ void window_start(const Segment* __restrict__ segs, const int32_t* __restrict__ leaf_start,
                                             int g0, int g1, Window& w) {
    w.nlo = w.nhi = 0;
    w.g = g0;
    window_load(segs, leaf_start, g1, w);
    window_load(segs, leaf_start, g1, w);
}

// Returns the tile's source count (0: the item's sources are exhausted);
// `guard` is set when a piece overlaps the targets [t0, t1) (a tile that holds
// the targets themselves).  The transaction bytes of each round are expected
// on `bar` by lane 0 before any lane issues its copy.
// With COPY false the tile is only passed over.
template <typename S4, int TILE, bool COPY>
__device__ __forceinline__ int pack_tile(const Segment* __restrict__ segs, const int32_t* __restrict__ leaf_start,
                                         int g1, Window& w, int t0, int t1, const S4* __restrict__ src, S4* dst,
                                         uint64_t* bar, bool& guard) {
    const int lane = threadIdx.x & 31;
    int count = 0;
    bool gd = false;
    while (count < TILE) {
        const int len = max(w.hi - w.lo, 0);
        int incl = len;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, incl, d);
            if (lane >= d) incl += y;
        }
        const int excl = incl - len;
        const int room = TILE - count;
        const int take = max(0, min(len, room - excl));
        const int total = __shfl_sync(0xffffffffu, incl, 31);
        const int placed = min(total, room);
        if (placed > 0) {
            if (COPY) {
                if (lane == 0) mbar_expect_tx(bar, uint32_t(placed) * uint32_t(sizeof(S4)));
                __syncwarp();
                if (take > 0) {
                    bulk_g2s(dst + count + excl, src + w.lo, uint32_t(take) * uint32_t(sizeof(S4)), bar);
                    if (w.lo < t1 && w.lo + take > t0) gd = true;
                }
            }
            w.lo += take;
            count += placed;
        }
        if (total <= room) {  // the window is used up
            if (w.g - 32 >= g1) break;  // and there is none after it
            window_load(segs, leaf_start, g1, w);
        }
    }
    if (COPY) guard = __any_sync(0xffffffffu, gd) != 0;
    return count;
}

// Sum over the L lanes of each group [L t, L t + L) of the warp (segmented
// tree of shuffles, L warp-uniform); the group's first lane (sub = 0) holds
// the sum.
template <typename T>
__device__ __forceinline__ T group_sum(T x, int sub, int L) {
    for (int off = 1; off < L; off <<= 1) {
        const T y = __shfl_down_sync(0xffffffffu, x, off);
        if (sub + off < L) x += y;
    }
    return x;
}

// Dynamic shared memory above the default limit has to be allowed, on every
// device that launches the kernel.
template <typename K>
inline cudaError_t allow_smem(K kernel, size_t bytes) {
    return bytes > 48 * 1024 ? cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(bytes))
                             : cudaSuccess;
}

}  // namespace fss
