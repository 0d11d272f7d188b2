// k_pairs.cu -- the FP32 pair engine shared by the direct sum, the near field
// and the far field (the FP64 engine is k_plane.cu), and the dispatch of both.
//
// A block works on one work item: the targets of one leaf (taken in chunks of
// CHUNK; the leaf's current particle range is read from leaf_start on the
// device, since particles are re-sorted into the leaves they have moved into)
// or an explicit target range (direct sum, a target cluster's interpolation
// points).  Its sources are a list of segments -- the particles of a run of
// leaves (range read at run time) or a fixed range -- packed back to back
// into tiles of kTile.  A tile belongs to one warp for all targets of the
// chunk, or to one warp for each of the 2 or 4 subsets of them that the item
// asks for (WorkItem::split): that warp brings it into its own landing buffer
// by bulk TMA copies (cp.async.bulk, no multicast; completion counted on its
// mbarrier), turns it into structure-of-arrays order, starts the copy of its
// next tile, and sums the tile for its targets.  Per pair (23 algorithmic
// flops):
//
//   d   = x_j - x_i
//   r2  = |d|^2           (= 2 (1 - x_i.x_j) on the unit sphere, no cancellation)
//   A  += w_j d / r2
//
// and afterwards u_i = -(1/2pi) x_i x A_i, since x_i x x_j = x_i x d and
// G(x_i, x_j) = 2 x_i x d / |d|^2.  A tile's FP32 sums are folded into a
// Kahan-compensated per-target total in the order of the tiles (each warp
// waits for its turn), so the result does not depend on the warps.
//
// Why whole tiles per warp and not 32 targets per warp: a warp's work no
// longer depends on which targets it has.  With one warp per 32 targets, the
// warps of a leaf of 78 particles left one of the SM's four partitions with a
// half-empty warp and one with none, and such leaves ran at 2.0e12 pairs/s
// where leaves of 128 ran at 2.45e12.  And a lane now takes two targets at a
// time, so that each source it loads serves both: in a loop of this
// instruction mix alone one target a lane takes 57 cycles per four sources
// and warp, two take 51 (20 packed FMA-pipe instructions are 40 cycles if
// nothing else is in the way, 4 reciprocals 32 of their own pipe).
#include <algorithm>

#include "pairs_common.cuh"

namespace fss {

// Quads per step of the pair loop, as measured: eight for two targets a lane
// (four: 163,842 particles 2,234 us a step instead of 2,197); four for one, the
// rest of an item's targets (eight: 40,962 particles with target clusters 377
// instead of 361); two with the stream function, whose loop is much the longer
// (eight: the sums of 163,842 particles 832 us instead of 690, with target
// clusters 434 instead of 330).
constexpr int unroll(bool psi, int targets) { return psi ? 2 : (targets == 1 ? 4 : 8); }
constexpr int kTile = kTileSources;
constexpr float kSelfR2 = 1e-30f;  // r^2 bias of the pair loop (a normal float; 1 / kSelfR2 finite)

// Sums of a tile in structure-of-arrays order (x[kTile], y, z, w, padded to a
// multiple of 4 sources with w = 0 at the origin: |x_i - 0|^2 = 1, no
// contribution) for NT targets of a lane (nt = minus their coordinates).  One
// 128-bit shared load brings a component of four sources; each pair of
// sources goes through the packed f32x2 pipe.  The self pair (and any source
// at the target's position) needs no select: r^2 starts from kSelfR2 = 1e-30
// inside the first FMA, so it gets 1 / r^2 = 1e30 and w 1e30 * (x_j - x_i) =
// 0; every other pair's r^2 (at least ~1e-12 between distinct particles on
// the unit sphere) is unchanged by the bias except when the exact d_x^2 falls
// on a rounding tie.  Only the stream function's log needs the guard (GUARD:
// tiles holding targets).  Quads q = q0, q0 + step, ... < nquad of the tile.
template <bool PSI, bool GUARD, int NT>
__device__ __forceinline__ void tile_pairs(const float* __restrict__ s, int nquad, int q0, int step,
                                           const float4 (&nt)[NT], float (&sx)[NT], float (&sy)[NT], float (&sz)[NT],
                                           float (&ap)[NT]) {
    const f2 eps = f2_pack(kSelfR2, kSelfR2);
    f2 ntx[NT], nty[NT], ntz[NT], ax[NT], ay[NT], az[NT];
#pragma unroll
    for (int k = 0; k < NT; k++) {
        ntx[k] = f2_pack(nt[k].x, nt[k].x);
        nty[k] = f2_pack(nt[k].y, nt[k].y);
        ntz[k] = f2_pack(nt[k].z, nt[k].z);
        ax[k] = ay[k] = az[k] = 0;
        ap[k] = 0.f;
    }
#pragma unroll(unroll(PSI, NT))
    for (int q = q0; q < nquad; q += step) {
        const float4 X = reinterpret_cast<const float4*>(s)[q];
        const float4 Y = reinterpret_cast<const float4*>(s + kTile)[q];
        const float4 Z = reinterpret_cast<const float4*>(s + 2 * kTile)[q];
        const float4 W = reinterpret_cast<const float4*>(s + 3 * kTile)[q];
        const f2 qx[2] = {f2_pack(X.x, X.y), f2_pack(X.z, X.w)};
        const f2 qy[2] = {f2_pack(Y.x, Y.y), f2_pack(Y.z, Y.w)};
        const f2 qz[2] = {f2_pack(Z.x, Z.y), f2_pack(Z.z, Z.w)};
        const f2 qw[2] = {f2_pack(W.x, W.y), f2_pack(W.z, W.w)};
#pragma unroll
        for (int h = 0; h < 2; h++)
#pragma unroll
            for (int k = 0; k < NT; k++) {
                const f2 dx = f2_add(qx[h], ntx[k]);
                const f2 dy = f2_add(qy[h], nty[k]);
                const f2 dz = f2_add(qz[h], ntz[k]);
                const f2 r2 = f2_fma(dz, dz, f2_fma(dy, dy, f2_fma(dx, dx, eps)));
                float r0, r1;
                f2_unpack(r2, r0, r1);
                const float i0 = rcp_fast(r0), i1 = rcp_fast(r1);
                const f2 sc = f2_mul(qw[h], f2_pack(i0, i1));
                ax[k] = f2_fma(sc, dx, ax[k]);
                ay[k] = f2_fma(sc, dy, ay[k]);
                az[k] = f2_fma(sc, dz, az[k]);
                if (PSI) {
                    float l0 = lg2_fast(r0), l1 = lg2_fast(r1);
                    if (GUARD) {
                        l0 = (r0 > kSelfR2) ? l0 : 0.f;
                        l1 = (r1 > kSelfR2) ? l1 : 0.f;
                    }
                    float w0, w1;
                    f2_unpack(qw[h], w0, w1);
                    ap[k] = fmaf(w0, l0, fmaf(w1, l1, ap[k]));
                }
            }
    }
#pragma unroll
    for (int k = 0; k < NT; k++) {
        float a0, a1;
        f2_unpack(ax[k], a0, a1);
        sx[k] = a0 + a1;
        f2_unpack(ay[k], a0, a1);
        sy[k] = a0 + a1;
        f2_unpack(az[k], a0, a1);
        sz[k] = a0 + a1;
    }
}

// A landed tile of `cnt` float4 sources into structure-of-arrays order, by
// one warp (lane L takes sources L, L + 32, ...: conflict-free), [cnt,
// 4 ceil(cnt / 4)) padded with zeros.
__device__ __forceinline__ void tile_to_soa(const float4* __restrict__ in, float* __restrict__ out, int cnt) {
    const int padded = (cnt + 3) & ~3;
#pragma unroll
    for (int k = 0; k < kTile / 32; k++) {
        const int j = (threadIdx.x & 31) + 32 * k;
        if (j < padded) {
            const float4 v = j < cnt ? in[j] : make_float4(0.f, 0.f, 0.f, 0.f);
            out[j] = v.x;
            out[kTile + j] = v.y;
            out[2 * kTile + j] = v.z;
            out[3 * kTile + j] = v.w;
        }
    }
}

__device__ __forceinline__ void kahan_add(float& sum, float& comp, float x) {
    const float y = x - comp;
    const float t = sum + y;
    comp = (t - sum) - y;
    sum = t;
}

// Turns of the warps at the totals, in the order of the tiles.
__device__ __forceinline__ int turn_load(const int* p) {
    int v;
    asm volatile("ld.acquire.cta.shared::cta.s32 %0, [%1];" : "=r"(v) : "r"(smem_addr(p)) : "memory");
    return v;
}
__device__ __forceinline__ void turn_store(int* p, int v) {
    asm volatile("st.release.cta.shared::cta.s32 [%0], %1;" ::"r"(smem_addr(p)), "r"(v) : "memory");
}

// Shared memory of a pair block.  A target's Kahan total: sums and
// corrections of x, y, z (and the log).
struct Total {
    float sx, sy, sz, cx, cy, cz;
};
template <int WARPS, bool PSI, int CHUNK>
struct PairSmem {
    float4 land[WARPS][kTile];
    float soa[WARPS][4 * kTile];
    Total total[CHUNK];
    float2 psi[PSI ? CHUNK : 1];
    uint64_t bar[WARPS];
    int turn[CHUNK / 32 + 1];  // per group of targets (the first of a pair): tiles folded into the totals
    int failed;                  // a wait gave up: the others need not wait out theirs
};

// One work item.  `phase` counts the warp's copies over all its items (the
// parity of its mbarrier).
template <int WARPS, bool PSI, int CHUNK>
__device__ __forceinline__ bool run_item(const WorkItem& it, const float4* __restrict__ src,
                                         const Segment* __restrict__ segs, const int32_t* __restrict__ leaf_start,
                                         double4* __restrict__ partials, int64_t pstride,
                                         PairSmem<WARPS, PSI, CHUNK>& sm, int& phase, int rotate, const PairCtl& ctl,
                                         bool hold) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    float4* land = sm.land[warp];
    float* soa = sm.soa[warp];
    int t0 = it.t0, nt = it.nt;
    if (it.leaf >= 0) {
        t0 = leaf_start[it.leaf] + it.t0;
        nt = leaf_start[it.leaf + 1] - t0;
        if (it.nt > 0) nt = min(nt, it.nt);
    }
    // the targets' groups of 32 in H subsets, each with `stride` warps that take
    // every stride-th tile; the warp's first tile rotates from item to item (the
    // warps of a block keep to their partitions of the SM)
    const int H = (it.split > 1 && WARPS % it.split == 0) ? it.split : 1;
    const int stride = WARPS / H, h = warp % H;
    const int mine = (warp / H + rotate) % stride;
    for (int c0 = 0; c0 < nt; c0 += CHUNK) {
        const int cn = min(CHUNK, nt - c0);
        // targets [32 g, 32 g + 32) of the chunk for g < full, one a lane, in
        // pairs of groups; each of the r left over gets L = 32 / r lanes, which
        // split a tile's quads between them and add their sums by shuffles
        const int full = cn >> 5, r = cn & 31;
        const int L = r > 0 ? 32 / r : 1;
        const int sub = lane % L, tl = lane / L;
        const int G = full + (r > 0 ? 1 : 0), ga = G * h / H, gb = G * (h + 1) / H;  // the warp's groups
        Window win;
        int pending = 0;  // sources on their way to `land`
        bool guard = false;
        bool mute = hold && c0 == 0 && mine == 0;  // test hook: no copy, no arrival for the first tile
        auto issue = [&](int skip) {
            bool none = false;
            for (int k = 0; k < skip && !none; k++)
                none = pack_tile<float4, kTile, false>(segs, leaf_start, it.g1, win, 0, 0, src, land, nullptr,
                                                       guard) == 0;
            pending = 0;
            if (none) return;
            if (mute) {
                pending = 1;
                mute = false;
                return;
            }
            pending = pack_tile<float4, kTile, true>(segs, leaf_start, it.g1, win, t0, t0 + nt, src, land,
                                                     &sm.bar[warp], guard);
            if (pending > 0 && lane == 0) mbar_arrive(&sm.bar[warp]);
        };
        if (ga < gb) {
            window_start(segs, leaf_start, it.g0, it.g1, win);
            issue(mine);
        }
        for (int i = tid; i < cn; i += 32 * WARPS) {
            sm.total[i] = Total{0, 0, 0, 0, 0, 0};
            if (PSI) sm.psi[i] = make_float2(0.f, 0.f);
        }
        if (tid <= CHUNK / 32) sm.turn[tid] = 0;
        __syncthreads();
        bool failed = false;
        for (int tile = mine; pending > 0; tile += stride) {
            const int cnt = pending;
            const bool gd = guard;
            if (!__all_sync(0xffffffffu, mbar_wait_bounded(&sm.bar[warp], uint32_t(phase) & 1, ctl.wait_ns))) {
                failed = true;
                break;
            }
            phase++;
            tile_to_soa(land, soa, cnt);
            __syncwarp();
            issue(stride - 1);  // the next tile on its way
            const int nq = (cnt + 3) >> 2;
            const float4* tgt = src + t0 + c0;
            // a unit of the targets (group g, or two groups) may be folded into the
            // totals once the tile before has been
            auto turn = [&](int g) {
                if (turn_load(&sm.turn[g]) != tile) {
                    const uint64_t since = global_timer_ns();
                    while (turn_load(&sm.turn[g]) != tile && !failed) {
                        __nanosleep(100);
                        failed = global_timer_ns() - since > ctl.wait_ns || turn_load(&sm.failed) != 0;
                    }
                }
                failed = __any_sync(0xffffffffu, failed) != 0;
            };
            auto next = [&](int g) {
                __syncwarp();
                if (lane == 0) turn_store(&sm.turn[g], tile + 1);
            };
            auto fold = [&](int i, float x, float y, float z, float p) {
                Total a = sm.total[i];
                kahan_add(a.sx, a.cx, x);
                kahan_add(a.sy, a.cy, y);
                kahan_add(a.sz, a.cz, z);
                sm.total[i] = a;
                if (PSI) {
                    float2 b = sm.psi[i];
                    kahan_add(b.x, b.y, p);
                    sm.psi[i] = b;
                }
            };
            const int gf = min(gb, full);
            int g = ga;
            for (; g + 2 <= gf && !failed; g += 2) {
                float4 x[2];
                float sx[2], sy[2], sz[2], sp[2];
#pragma unroll
                for (int k = 0; k < 2; k++) {
                    const float4 v = tgt[32 * (g + k) + lane];
                    x[k] = make_float4(-v.x, -v.y, -v.z, 0.f);
                }
                if (PSI && gd)
                    tile_pairs<PSI, true, 2>(soa, nq, 0, 1, x, sx, sy, sz, sp);
                else
                    tile_pairs<PSI, false, 2>(soa, nq, 0, 1, x, sx, sy, sz, sp);
                turn(g);
                if (failed) break;
#pragma unroll
                for (int k = 0; k < 2; k++) fold(32 * (g + k) + lane, sx[k], sy[k], sz[k], sp[k]);
                next(g);
            }
            if (g < gf && !failed) {
                float4 x[1];
                float sx[1], sy[1], sz[1], sp[1];
                const float4 v = tgt[32 * g + lane];
                x[0] = make_float4(-v.x, -v.y, -v.z, 0.f);
                if (PSI && gd)
                    tile_pairs<PSI, true, 1>(soa, nq, 0, 1, x, sx, sy, sz, sp);
                else
                    tile_pairs<PSI, false, 1>(soa, nq, 0, 1, x, sx, sy, sz, sp);
                turn(g);
                if (!failed) {
                    fold(32 * g + lane, sx[0], sy[0], sz[0], sp[0]);
                    next(g);
                }
            }
            if (gb > full && !failed) {
                float4 x[1];
                float sx[1], sy[1], sz[1], sp[1];
                const float4 v = tgt[32 * full + min(tl, r - 1)];
                x[0] = make_float4(-v.x, -v.y, -v.z, 0.f);
                if (PSI && gd)
                    tile_pairs<PSI, true, 1>(soa, nq, sub, L, x, sx, sy, sz, sp);
                else
                    tile_pairs<PSI, false, 1>(soa, nq, sub, L, x, sx, sy, sz, sp);
                sx[0] = group_sum(sx[0], sub, L);
                sy[0] = group_sum(sy[0], sub, L);
                sz[0] = group_sum(sz[0], sub, L);
                if (PSI) sp[0] = group_sum(sp[0], sub, L);
                turn(full);
                if (!failed) {
                    if (sub == 0 && tl < r) fold(32 * full + tl, sx[0], sy[0], sz[0], sp[0]);
                    next(full);
                }
            }
            if (failed) break;
            __syncwarp();  // the tile is used up before the next one takes its place
        }
        if (failed) {
            // no bulk copy may still be landing in this block's shared memory
            // when it exits: the warp waits (bounded) for its own
            if (lane == 0) turn_store(&sm.failed, 1);
            if (pending > 0) mbar_wait_bounded(&sm.bar[warp], uint32_t(phase) & 1, ctl.wait_ns);
        }
        if (__syncthreads_or(failed)) return false;
        for (int i = tid; i < cn; i += 32 * WARPS) {
            const Total a = sm.total[i];
            double4 o = make_double4(double(a.sx) - double(a.cx), double(a.sy) - double(a.cy),
                                     double(a.sz) - double(a.cz), 0.0);
            if (PSI) o.w = double(sm.psi[i].x) - double(sm.psi[i].y);
            partials[int64_t(it.part) * pstride + t0 + c0 + i] = o;
        }
        __syncthreads();
    }
    return true;
}

template <int WARPS, bool PSI, int CHUNK>
__device__ __forceinline__ void init_block(PairSmem<WARPS, PSI, CHUNK>& sm) {
    if (threadIdx.x < WARPS) mbar_init(&sm.bar[threadIdx.x], 1);
    if (threadIdx.x == 0) sm.failed = 0;
    mbar_init_fence();
    __syncthreads();
}

// Twenty warps per SM: 96 registers a thread (24 at 80 are no faster).
constexpr int blocks_per_sm(int threads) { return 640 / threads; }

// One block per work item.
template <int THREADS, bool PSI, int CHUNK>
__global__ void __launch_bounds__(THREADS, blocks_per_sm(THREADS))
    k_pairs(const float4* __restrict__ src, const Segment* __restrict__ segs, const int32_t* __restrict__ leaf_start,
            const WorkItem* __restrict__ items, double4* __restrict__ partials, int64_t pstride,
            int* __restrict__ err, const PairCtl ctl) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    auto& sm = *reinterpret_cast<PairSmem<THREADS / 32, PSI, CHUNK>*>(smem_raw);
    init_block(sm);
    int phase = 0;
    const WorkItem it = items[blockIdx.x];
    if (!run_item<THREADS / 32, PSI, CHUNK>(it, src, segs, leaf_start, partials, pstride, sm, phase, int(blockIdx.x), ctl,
                                            int(blockIdx.x) == ctl.hold_block) &&
        threadIdx.x == 0)
        set_error(err, kErrTimeout);
}

// Persistent blocks pulling work items from one global queue (reset to 0
// before every launch); the copies' phases run on from item to item.
template <int THREADS, int CHUNK>
__global__ void __launch_bounds__(THREADS, blocks_per_sm(THREADS))
    k_pairs_persistent(const float4* __restrict__ src, const Segment* __restrict__ segs,
                       const int32_t* __restrict__ leaf_start, const WorkItem* __restrict__ items, int nitems,
                       int* __restrict__ queue, double4* __restrict__ partials, int64_t pstride,
                       int* __restrict__ err, const PairCtl ctl) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ int next_item;
    auto& sm = *reinterpret_cast<PairSmem<THREADS / 32, false, CHUNK>*>(smem_raw);
    init_block(sm);
    int phase = 0;
    for (;;) {
        if (threadIdx.x == 0) next_item = atomicAdd(queue, 1);
        __syncthreads();
        const int item = next_item;
        __syncthreads();
        if (item >= nitems) return;
        const WorkItem it = items[item];
        if (!run_item<THREADS / 32, false, CHUNK>(it, src, segs, leaf_start, partials, pstride, sm, phase, item, ctl,
                                                 false)) {
            if (threadIdx.x == 0) set_error(err, kErrTimeout);
            return;
        }
    }
}

// ---------------------------------------------------------------- dispatch

// Targets of one pass (pass_targets): leaves, target clusters and small items
// have at most kSmallChunk; only where some have more do their totals take the
// larger share of an SM's memory from the L1 cache, which the concurrent kernels
// of a step use: 163,842 particles with target clusters 1,448 us per step, 1,459
// with the larger one; 300,001 in leaves of 234, which then take two passes,
// 2,838 and 2,675.

template <int WARPS, bool PSI, int CHUNK>
static cudaError_t run_pairs(cudaStream_t st, int nitems, const void* src, const Segment* segs,
                             const int32_t* leaf_start, const WorkItem* items, double4* partials, int64_t pstride,
                             int* err, PairCtl ctl) {
    constexpr size_t smem = sizeof(PairSmem<WARPS, PSI, CHUNK>);
    const cudaError_t e = allow_smem(k_pairs<32 * WARPS, PSI, CHUNK>, smem);
    if (e != cudaSuccess) return e;
    k_pairs<32 * WARPS, PSI, CHUNK><<<nitems, 32 * WARPS, smem, st>>>(
        static_cast<const float4*>(src), segs, leaf_start, items, partials, pstride, err, ctl);
    return cudaGetLastError();
}

PairShape pairs_shape(int threads) {
    PairShape s;
    if (threads == 192 || threads == 224 || threads == 288) s.threads = threads;
    return s;
}

// FP32: four warps when all items run at once anyway (740 such blocks fit; us
// per RK4 step of 100 clusters in 4 parts 166, with two warps 186), else two:
// smaller pieces of work beside the leaves' launch (420 in 4 parts 394, with four
// warps 416; 6,820 4,032 and 4,126).
PairShape cluster_shape(bool fp64, int64_t items) {
    PairShape s;
    if (!fp64 && items >= 740) s.warps = 2;
    s.max_targets = kMaxK;
    return s;
}

template <bool PSI, int CHUNK>
static cudaError_t dispatch(cudaStream_t st, int warps, int nitems, const void* src, const Segment* segs,
                            const int32_t* leaf_start, const WorkItem* items, double4* partials, int64_t pstride,
                            int* err, PairCtl ctl) {
    auto run = warps == 2 ? run_pairs<2, PSI, CHUNK> : run_pairs<4, PSI, CHUNK>;
    return run(st, nitems, src, segs, leaf_start, items, partials, pstride, err, ctl);
}

cudaError_t launch_pairs(cudaStream_t st, bool fp64, bool psi, PairShape shape, int nitems, const void* src,
                         const Segment* segs, const int32_t* leaf_start, const WorkItem* items,
                         double4* partials, int64_t pstride, int* err, PairCtl ctl) {
    if (nitems == 0) return cudaSuccess;
    if (fp64)
        return launch_plane_pairs(st, psi, nitems, src, segs, leaf_start, items, partials, pstride, err, ctl);
    auto run = pass_targets(shape.max_targets) == kSmallChunk ? (psi ? dispatch<true, kSmallChunk> : dispatch<false, kSmallChunk>)
                                                              : (psi ? dispatch<true, kLargeChunk> : dispatch<false, kLargeChunk>);
    return run(st, shape.warps, nitems, src, segs, leaf_start, items, partials, pstride, err, ctl);
}

cudaError_t launch_pairs_persistent(cudaStream_t st, int nitems, const void* src, const Segment* segs,
                                    const int32_t* leaf_start, const WorkItem* items, int* queue,
                                    double4* partials, int64_t pstride, int* err, int blocks, PairCtl ctl) {
    constexpr size_t smem = sizeof(PairSmem<kPersistentThreads / 32, false, kSmallChunk>);
    if (nitems == 0) return cudaSuccess;
    const cudaError_t e = allow_smem(k_pairs_persistent<kPersistentThreads, kSmallChunk>, smem);
    if (e != cudaSuccess) return e;
    k_pairs_persistent<kPersistentThreads, kSmallChunk><<<blocks, kPersistentThreads, smem, st>>>(
        static_cast<const float4*>(src), segs, leaf_start, items, nitems, queue, partials, pstride, err, ctl);
    return cudaGetLastError();
}

int persistent_blocks_per_sm() {
    constexpr size_t smem = sizeof(PairSmem<kPersistentThreads / 32, false, kSmallChunk>);
    int nb = 0;
    allow_smem(k_pairs_persistent<kPersistentThreads, kSmallChunk>, smem);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_pairs_persistent<kPersistentThreads, kSmallChunk>, kPersistentThreads,
                                                  smem);
    return nb > 0 ? nb : 1;
}

}  // namespace fss
