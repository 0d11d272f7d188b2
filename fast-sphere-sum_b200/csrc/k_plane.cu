// k_plane.cu -- the FP64 pair engine: direct sum, near field and far field,
// summed in the plane.
//
// A block works on one work item: the targets of one leaf (taken in chunks,
// chunk_targets; the leaf's current particle range is read from leaf_start on
// the device, since particles are re-sorted into the leaves they have moved
// into) or an explicit target range (direct sum, a target cluster's
// interpolation points).  Its sources are a list of segments -- the particles
// of a run of leaves (range read at run time) or a fixed range -- packed back
// to back into shared-memory tiles by bulk TMA copies (cp.async.bulk, no
// multicast) whose completion is counted on the tile slot's mbarrier.
//
// With c near the targets, e1, e2 orthonormal to it and the stereographic
// coordinates from -c,
//
//   xi(x) = (x.e1, x.e2) / (1 + x.c),    rho = |xi|^2,
//   |x_j - x_i|^2 = 4 |xi_j - xi_i|^2 / ((1 + rho_i)(1 + rho_j)),
//
// the sum A = sum_j w_j (x_j - x_i) / |x_j - x_i|^2 that the velocity
// u_i = -(1/2pi) x_i x A and the target clusters' interpolants need is, by
// the gradient of log|x_j - x_i|^2 along the sphere (conformal map) and
// (x_j - x_i).x_i = -|x_j - x_i|^2 / 2 across it,
//
//   B  = sum_j w_j (xi_j - xi_i) / |xi_j - xi_i|^2        (the pair loop)
//   P  = B + W xi_i / (1 + rho_i),   W = sum_j w_j
//   A  = (1 + rho_i)/2 (P_1 e1 + P_2 e2) - (P.xi_i)(xi_i.e + c) - (W/2) x_i
//
// so that a pair costs 10 FP64 operations (2 differences, 2 for r^2, 4 for
// w / r^2, 2 accumulations) where differences in space cost 14; everything
// else is done once per source and chunk (about 40 operations) or once per
// target.  The map keeps the relative precision of x - c near the targets, so
// neighbours' differences carry the rounding of the positions and no more.
//
// The map holds on the unit sphere alone and serves targets on c's side of it
// (kMinCos).  What it does not serve is summed in space, at 14 operations a
// pair: a warp's share of a tile with a source off the sphere (kOnSphere), and
// every share for a chunk with a target off it or with targets all over it
// (a tree evaluated at other positions than its own: 163,842 particles 1.40 ms,
// where a pass over the sources around each group of targets took 4.31).
//
// Bound by the FP64 pipe, 80% busy (20 of the 27 cycles that a pair takes a
// warp).  Per right-hand side, before and now: treecode of 163,842 particles
// (n = 8, theta = 0.7; 1.29e9 lane pairs) 1.347 and 0.918 ms; direct sum of
// 20,011 particles 0.403 and 0.33 ms; 40,962 particles with the stream
// function 1.18 and 0.48 ms.
// The FP32 engine (k_pairs.cu) sums in space.
#include <algorithm>

#include "pairs_common.cuh"

namespace fss {

constexpr int kUnroll = 2;       // units per step of the pair loop
constexpr int kDepth = 2;        // ring depth (tiles in flight)
constexpr int kTile = tile_capacity(true);
constexpr double kMinCos = 0.2;  // the plane serves targets with x.c above this
constexpr int kSlots = 32 * (kMaxFull + 1);  // accumulator slots of a warp

// What the guarded pair loop adds to r^2, so that a source at the target's
// position (r^2 = 0) has a finite reciprocal that multiplies a zero
// difference; far below any other r^2.
constexpr double kSelfR2 = 1e-200;
// Where a tile's padding (w = 0) and a source at the antipode -c lie: where
// they add nothing.
constexpr double kFarAway = 1e100;

// | |x|^2 - 1 | of a point on the unit sphere: the rounding of a normalised
// position is below 2^-50.
constexpr double kOnSphere = 0x1p-48;
__device__ __forceinline__ double norm2(double x, double y, double z) {
    return __fma_rn(z, z, __fma_rn(y, y, __dmul_rn(x, x)));
}
__device__ __forceinline__ bool on_sphere(double x, double y, double z) {
    return fabs(norm2(x, y, z) - 1.0) <= kOnSphere;  // false for a non-finite position
}

// The plane of a chunk of targets, in shared memory.
struct PlaneShared {
    double c[3], e1[3], e2[3];
    int flat;  // it serves them
};
struct Plane {
    double c[3], a[3], b[3];
    __device__ __forceinline__ void load(const PlaneShared& s) {
#pragma unroll
        for (int k = 0; k < 3; k++) {
            c[k] = s.c[k];
            a[k] = s.e1[k];
            b[k] = s.e2[k];
        }
    }
    __device__ __forceinline__ bool serves(double x, double y, double z) const {
        return x * c[0] + y * c[1] + z * c[2] > kMinCos;
    }
};

// Stereographic coordinates of a point near the unit sphere, put on it first
// (two Newton steps for 1 / |x|: a position rounded to few digits must not be
// moved along the sphere by its distance from it).  With t = x - c on c's
// side, 1 + x.c = (4 - |t|^2) / 2; with t = x + c on the other, |t|^2 / 2 (and
// x.e = t.e either way); close to the antipode -c, where t's radial part is
// rounding, |t|^2 = 2 (1 - sqrt(1 - q)) with q = (t.e1)^2 + (t.e2)^2.
// Explicitly rounded operations: a target and the same point as a source must
// map to the same bits.
__device__ __forceinline__ void plane_map(const Plane& p, double x, double y, double z, double& u, double& v) {
    const double nn = norm2(x, y, z);
    double n = __fma_rn(-0.5, nn, 1.5);
    n = __dmul_rn(n, __fma_rn(__dmul_rn(-0.5, nn), __dmul_rn(n, n), 1.5));
    x = __dmul_rn(x, n);
    y = __dmul_rn(y, n);
    z = __dmul_rn(z, n);
    const double dc = __fma_rn(z, p.c[2], __fma_rn(y, p.c[1], __dmul_rn(x, p.c[0])));
    const double s = -copysign(1.0, dc);
    const double tx = __fma_rn(s, p.c[0], x), ty = __fma_rn(s, p.c[1], y), tz = __fma_rn(s, p.c[2], z);
    const double tt = __fma_rn(tz, tz, __fma_rn(ty, ty, __dmul_rn(tx, tx)));
    const bool far = s > 0.0;
    const double a = __fma_rn(tz, p.a[2], __fma_rn(ty, p.a[1], __dmul_rn(tx, p.a[0])));
    const double b = __fma_rn(tz, p.b[2], __fma_rn(ty, p.b[1], __dmul_rn(tx, p.b[0])));
    if (far && tt < 1e-2) {
        const double q = a * a + b * b;
        const double k = (1.0 + sqrt(1.0 - q)) / q;
        const bool away = q > 1e-60;
        u = away ? a * k : kFarAway;
        v = away ? b * k : 0.0;
        return;
    }
    const double k = rcp_fast(__dmul_rn(0.5, far ? tt : __dsub_rn(4.0, tt)));
    u = __dmul_rn(a, k);
    v = __dmul_rn(b, k);
}

// The plane around (x, y, z): c its direction, e1 and e2 by the branchless
// construction of Duff et al., "Building an orthonormal basis, revisited"
// (JCGT 6, 2017).  Without a direction it is the pole.
__device__ __forceinline__ void plane_around(double x, double y, double z, PlaneShared& s) {
    const double nn = x * x + y * y + z * z;
    const double r = rsqrt(nn);
    const bool ok = nn > 0.0 && nn < 1e300;
    x = ok ? x * r : 0.0;
    y = ok ? y * r : 0.0;
    z = ok ? z * r : 1.0;
    const double sg = copysign(1.0, z), a = -1.0 / (sg + z), b = x * y * a;
    s.c[0] = x;
    s.c[1] = y;
    s.c[2] = z;
    s.e1[0] = 1.0 + sg * x * x * a;
    s.e1[1] = sg * b;
    s.e1[2] = -sg * x;
    s.e2[0] = b;
    s.e2[1] = sg + y * y * a;
    s.e2[2] = -y;
}

// A lane's accumulators, one slot per target.
struct alignas(16) Acc {
    double u, v;
};
// The same for the sources summed in space: their share of A.
struct Acc3 {
    double x, y, z;
};

// log2 of r2 (positive, finite) beside its reciprocal's approximation y: y
// rounded to 5 mantissa bits, yt, makes r2 yt = 1 + r with |r| < 2^-6 and no
// rounding, and log2 r2 = log2(1 + r) - log2 yt, the first a Taylor
// polynomial of degree 8 (the term after it is below 2^-56), the second the
// exponent of yt and log2(1 + i/32) of its 5 bits from the table `lg`
// (P. T. P. Tang's table-driven logarithm, ACM TOMS 16, 1990, with a
// reciprocal in place of a division as in W. F. Wong and E. Goto, IEEE Trans.
// Computers 43, 1994).  About 12 FP64 operations where log2() took 75: the
// sums with the stream function of 40,962 particles 1.18 ms with
// log2(), 0.48 ms with this.
__device__ __forceinline__ double log2_beside(double r2, double y, const double* __restrict__ lg) {
    const int t = (__double2hiint(y) + 0x4000) & ~0x7fff;
    const double r = fma(r2, __hiloint2double(t, 0), -1.0);
    constexpr double c = 1.4426950408889634;  // 1 / ln 2
    double p = fma(r, -c / 8, c / 7);
    p = fma(r, p, -c / 6);
    p = fma(r, p, c / 5);
    p = fma(r, p, -c / 4);
    p = fma(r, p, c / 3);
    p = fma(r, p, -c / 2);
    p = fma(r, p, c);
    return fma(r, p, double(1023 - (t >> 20)) - lg[(t >> 15) & 31]);
}

// Pairs of NT targets of a lane with units (two sources, one 128-bit load per
// component) q0, q0 + step, ... < q1 of mapped sources (arrays u, v, w of
// SHARE entries, padded to whole units with w = 0).  A source at a target's
// position must add nothing, also not to W.  GUARD (the tiles known to hold
// the targets themselves): a bias on r^2 keeps its reciprocal finite, and its
// w is summed into wz as (w / r^2) times the bias -- exact for it, nothing for
// any other source.  Without GUARD its reciprocal is infinite and the sums
// come out NaN, for which the caller takes the sources again, guarded.
//
// The reciprocal is the hardware approximation y of 1 / r^2 (relative error
// e < 2^-18) refined by y (1 + e + e^2), error e^3 < 2^-54, folded into the
// product with w.
template <bool PSI, bool GUARD, int SHARE, int NT>
__device__ __forceinline__ void plane_pairs(const double* __restrict__ s, int q0, int q1, int step,
                                            const double2 (&t)[NT], double (&bu)[NT], double (&bv)[NT],
                                            double (&wz)[NT], double (&ap)[NT], const double* __restrict__ lg) {
#pragma unroll
    for (int k = 0; k < NT; k++) bu[k] = bv[k] = wz[k] = ap[k] = 0.0;
#pragma unroll(PSI ? 1 : (NT == 1 ? 4 : kUnroll))
    for (int q = q0; q < q1; q += step) {
        const double2 U = reinterpret_cast<const double2*>(s)[q];
        const double2 V = reinterpret_cast<const double2*>(s + SHARE)[q];
        const double2 W = reinterpret_cast<const double2*>(s + 2 * SHARE)[q];
        const double qu[2] = {U.x, U.y}, qv[2] = {V.x, V.y}, qw[2] = {W.x, W.y};
#pragma unroll
        for (int h = 0; h < 2; h++)
#pragma unroll
            for (int k = 0; k < NT; k++) {
                const double du = qu[h] - t[k].x, dv = qv[h] - t[k].y;
                const double r2 = fma(dv, dv, GUARD ? fma(du, du, kSelfR2) : du * du);
                const double y = rcp_seed(r2);
                const double e = fma(-r2, y, 1.0);
                const double wy = qw[h] * y;
                const double sc = fma(wy, fma(e, e, e), wy);
                bu[k] = fma(sc, du, bu[k]);
                bv[k] = fma(sc, dv, bv[k]);
                if (GUARD) wz[k] = fma(sc, kSelfR2, wz[k]);
                if (PSI) {
                    double l = log2_beside(r2, y, lg);
                    if (GUARD) l = (r2 > kSelfR2) ? l : 0.0;
                    ap[k] = fma(qw[h], l, ap[k]);
                }
            }
    }
}

// A warp's share of a tile for its lanes' NT targets (positions tpos[32 k]),
// added to the lane's accumulators.
template <bool PSI, int SHARE, int NT>
__device__ __forceinline__ void plane_fold(const double* __restrict__ share, int q0, int q1, int step, bool guard,
                                           const double2* tpos, Acc* acc, double* accp, double* wz,
                                           const double* lg) {
    const int lane = threadIdx.x & 31;
    double2 t[NT];
    double bu[NT], bv[NT], bz[NT], bp[NT];
#pragma unroll
    for (int k = 0; k < NT; k++) t[k] = tpos[32 * k];
    if (!guard) {
        plane_pairs<PSI, false, SHARE, NT>(share, q0, q1, step, t, bu, bv, bz, bp, lg);
        bool bad = false;
#pragma unroll
        for (int k = 0; k < NT; k++) bad |= !(bu[k] - bu[k] == 0.0) || !(bv[k] - bv[k] == 0.0);
        guard = __any_sync(0xffffffffu, bad);  // a source at a target's position (or a non-finite one)
    }
    if (guard) plane_pairs<PSI, true, SHARE, NT>(share, q0, q1, step, t, bu, bv, bz, bp, lg);
#pragma unroll
    for (int k = 0; k < NT; k++) {
        Acc& a = acc[32 * k + lane];
        a.u += bu[k];
        a.v += bv[k];
        if (PSI) accp[32 * k + lane] += bp[k];
        if (guard) wz[32 * k + lane] += bz[k];
    }
}

// Pairs of NT targets t of a lane with sources j0, j0 + step, ... < n as they
// landed, in space: A = sum w_j d / |d|^2, d = x_j - x_i, exact for neighbours,
// at any radius.  A source at the target's position adds nothing: r^2 starts
// from kSelfR2, so that its reciprocal is finite and multiplies d = 0.
template <bool PSI, int NT>
__device__ __forceinline__ void space_pairs(const double4* __restrict__ s, int j0, int n, int step,
                                            const double4 (&t)[NT], Acc3 (&a)[NT], double (&ap)[NT],
                                            const double* __restrict__ lg) {
#pragma unroll
    for (int k = 0; k < NT; k++) {
        a[k] = Acc3{};
        ap[k] = 0.0;
    }
#pragma unroll(PSI ? 1 : 2)
    for (int j = j0; j < n; j += step) {
        const double4 q = s[j];
#pragma unroll
        for (int k = 0; k < NT; k++) {
            const double dx = q.x - t[k].x, dy = q.y - t[k].y, dz = q.z - t[k].z;
            const double r2 = fma(dz, dz, fma(dy, dy, fma(dx, dx, kSelfR2)));
            const double sc = q.w * rcp_fast(r2);
            a[k].x = fma(sc, dx, a[k].x);
            a[k].y = fma(sc, dy, a[k].y);
            a[k].z = fma(sc, dz, a[k].z);
            if (PSI) {
                const double l = log2_beside(r2, rcp_seed(r2), lg);
                ap[k] = fma(q.w, (r2 > kSelfR2) ? l : 0.0, ap[k]);
            }
        }
    }
}

// A warp's share of a tile for its lanes' NT targets (tgt[32 k]) in space,
// added to the lane's accumulators.
template <bool PSI, int NT>
__device__ __forceinline__ void space_fold(const double4* __restrict__ share, int j0, int n, int step,
                                           const double4* __restrict__ tgt, Acc3* acc, double* accp,
                                           const double* lg) {
    const int lane = threadIdx.x & 31;
    double4 t[NT];
    Acc3 a[NT];
    double ap[NT];
#pragma unroll
    for (int k = 0; k < NT; k++) t[k] = tgt[32 * k];
    space_pairs<PSI, NT>(share, j0, n, step, t, a, ap, lg);
#pragma unroll
    for (int k = 0; k < NT; k++) {
        Acc3& o = acc[32 * k + lane];
        o.x += a[k].x;
        o.y += a[k].y;
        o.z += a[k].z;
        if (PSI) accp[32 * k + lane] += ap[k];
    }
}

// A warp's share of a landed tile -- n sources from `in` -- mapped to the
// plane (lane L takes sources L, L + 32, ...: conflict-free) into the warp's
// own arrays u, v, w of SHARE entries, padded to whole units with w = 0; the
// lane's sums of w and w log2(1 + rho) added to wsum and lsum.  False when a
// source is not on the sphere: the share is to be summed in space (and
// nothing is added).
template <bool PSI, int SHARE>
__device__ __forceinline__ bool map_share(const double4* __restrict__ in, double* __restrict__ out, int n,
                                          const Plane& p, double& wsum, double& lsum) {
    const int lane = threadIdx.x & 31;
    const int padded = (n + 1) & ~1;
    double ws = 0, ls = 0;
    bool flat = true;
#pragma unroll 2
    for (int j = lane; j < padded; j += 32) {
        double u = kFarAway, v = 0, w = 0;
        if (j < n) {
            const double4 q = in[j];
            flat = flat && on_sphere(q.x, q.y, q.z);
            plane_map(p, q.x, q.y, q.z, u, v);
            w = q.w;
        }
        out[j] = u;
        out[SHARE + j] = v;
        out[2 * SHARE + j] = w;
        ws += w;
        if (PSI) ls += w * lg2_fast(fma(v, v, fma(u, u, 1.0)));
    }
    if (!__all_sync(0xffffffffu, flat)) return false;
    wsum += ws;
    if (PSI) lsum += ls;
    return true;
}

// Tile header written by warp 0 before the slot's arrive (every warp reads it
// after the slot's phase completes).
struct SlotHdr {
    int count, guard;
};

struct RingState {
    int issued, taken;  // tiles, over all chunks
    bool failed;
};

// A target's A (and its log2 sum) from the sums in the plane.
template <bool PSI>
__device__ __forceinline__ double4 target_sum(const PlaneShared& ps, double wtot, double ltot, double x, double y, double z, double tu, double tv,
                                              double bu, double bv, double bp, double wz) {
    const double u = tu, v = tv, rho = u * u + v * v;
    const double W = wtot - wz, f = W / (1.0 + rho);
    const double p1 = bu + f * u, p2 = bv + f * v;
    const double g = 0.5 * (1.0 + rho), h = p1 * u + p2 * v;
    const double k1 = g * p1 - h * u, k2 = g * p2 - h * v, kx = 0.5 * W;
    double4 o;
    o.x = k1 * ps.e1[0] + k2 * ps.e2[0] - h * ps.c[0] - kx * x;
    o.y = k1 * ps.e1[1] + k2 * ps.e2[1] - h * ps.c[1] - kx * y;
    o.z = k1 * ps.e1[2] + k2 * ps.e2[2] - h * ps.c[2] - kx * z;
    o.w = 0.0;
    if (PSI)  // log2 |x_j - x_i|^2 = log2 |xi_j - xi_i|^2 + 2 - log2(1 + rho_i) - log2(1 + rho_j)
        o.w = bp + W * (2.0 - log2(1.0 + rho)) - (ltot - wz * lg2_fast(fma(tv, tv, fma(tu, tu, 1.0))));
    return o;
}

// Shared memory of a pair block: the landing ring (kDepth tiles as copied),
// and each warp's mapped share of a tile, accumulators and sums over its
// sources; the targets' plane coordinates.
template <int WARPS, bool PSI>
struct PairSmem {
    static constexpr int kShare = (kTile / 2 + WARPS - 1) / WARPS * 2;
    double4 ring[kDepth * kTile];
    double mapped[WARPS * 3 * kShare];
    Acc acc[WARPS * kSlots];
    Acc3 acc3[WARPS * kSlots];
    double2 tpos[kSlots];
    double wz[WARPS * kSlots];
    double accp[PSI ? WARPS * kSlots : 1];
    double wsum[WARPS], lsum[WARPS];
    double lg[PSI ? 32 : 1];  // log2(1 + i/32)
};
struct PairBars {
    uint64_t *full, *empty;
    SlotHdr* hdr;
    PlaneShared* ps;
};

// One work item: every chunk of targets against every tile of its segments.
// Warp 0 packs and issues the tiles, one ahead of the one in use.  Every warp
// maps its share of a landed tile to the plane, releases the slot through
// empty (a share summed in space is read from the slot, which is released
// after), and takes its share for all targets of the chunk: cn >> 5 targets a
// lane (a source loaded serves them all) and, for the r = cn & 31 left over,
// L = 32 / r lanes a target, which split the share between them.  So the
// warps' work is equal whatever the count of targets (one warp per 32 targets
// left the SM's quarters unequally loaded: leaves of 78 particles ran at 62%
// of the rate of leaves of 128), and no warp waits for another's mapping.
// The warps' sums are added at the end of the chunk.
template <int WARPS, bool PSI>
__device__ __forceinline__ void run_item(const WorkItem& it, const double4* __restrict__ src,
                                         const Segment* __restrict__ segs, const int32_t* __restrict__ leaf_start,
                                         double4* __restrict__ partials, int64_t pstride,
                                         PairSmem<WARPS, PSI>& sm, const PairBars& br, RingState& rs,
                                         const PairCtl& ctl, bool hold) {
    constexpr int SHARE = PairSmem<WARPS, PSI>::kShare;
    constexpr int UNIT = 2;  // sources per step of a lane
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    PlaneShared* ps = br.ps;
    int t0 = it.t0, nt = it.nt;
    if (it.leaf >= 0) {
        t0 = leaf_start[it.leaf];
        nt = leaf_start[it.leaf + 1] - t0;
    }
    const int chunk = chunk_targets(nt);
    for (int c0 = 0; c0 < nt; c0 += chunk) {
        const int cn = min(chunk, nt - c0);
        const int full = cn >> 5, r = cn & 31;
        const int L = r > 0 ? 32 / r : 1;
        // warp 0: the next tile into its slot (an empty one ends the chunk),
        // once every warp has mapped the tile before it there
        Window win;
        bool packed = false;  // the empty tile has been issued
        auto issue = [&]() {
            const int slot = rs.issued % kDepth;
            bool ok = true;
            if (rs.issued >= kDepth)
                ok = mbar_wait_bounded(&br.empty[slot], uint32_t((rs.issued / kDepth) - 1) & 1, ctl.wait_ns);
            if (!__all_sync(0xffffffffu, ok)) {
                rs.failed = true;
                return;
            }
            int cnt = 1;
            if (hold && rs.issued == 0) {
                // test hook: the first tile is neither copied nor signalled
                if (lane == 0) br.hdr[slot].count = cnt;
            } else {
                bool gd = false;
                cnt = pack_tile<double4, kTile, true>(segs, leaf_start, it.g1, win, t0, t0 + nt, src, sm.ring + slot * kTile,
                                          &br.full[slot], gd);
                if (lane == 0) {
                    br.hdr[slot].count = cnt;
                    br.hdr[slot].guard = gd ? 1 : 0;
                    mbar_arrive(&br.full[slot]);
                }
            }
            __syncwarp();
            packed = cnt == 0;
            rs.issued++;
        };
        if (warp == 0) {
            window_start(segs, leaf_start, it.g0, it.g1, win);
            issue();
        } else if (warp == 1) {
            // c: the direction of the chunk's targets' mean
            double mx = 0, my = 0, mz = 0;
            for (int i = lane; i < cn; i += 32) {
                const double4 v = src[t0 + c0 + i];
                mx += v.x;
                my += v.y;
                mz += v.z;
            }
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) {
                mx += __shfl_xor_sync(0xffffffffu, mx, off);
                my += __shfl_xor_sync(0xffffffffu, my, off);
                mz += __shfl_xor_sync(0xffffffffu, mz, off);
            }
            if (lane == 0) {
                plane_around(mx, my, mz, *ps);
                ps->flat = 1;
            }
        }
        Acc* acc = sm.acc + warp * kSlots;
        Acc3* acc3 = sm.acc3 + warp * kSlots;
        double* accp = PSI ? sm.accp + warp * kSlots : sm.accp;
        double* wz = sm.wz + warp * kSlots;
        double* mapped = sm.mapped + warp * 3 * SHARE;
        for (int k = lane; k < 32 * (full + 1); k += 32) {
            acc[k] = Acc{};
            acc3[k] = Acc3{};
            wz[k] = 0;
            if (PSI) accp[k] = 0.0;
        }
        __syncthreads();
        {
            Plane plane;
            plane.load(*ps);
            for (int i = tid; i < cn; i += 32 * WARPS) {
                const double4 v = src[t0 + c0 + i];
                double2 p;
                plane_map(plane, v.x, v.y, v.z, p.x, p.y);
                sm.tpos[i] = p;
                if (!on_sphere(v.x, v.y, v.z) || !plane.serves(v.x, v.y, v.z)) ps->flat = 0;
            }
        }
        __syncthreads();
        const bool flat = ps->flat != 0;
        double wsum = 0, lsum = 0;
        while (!rs.failed) {
            if (warp == 0 && !packed) {
                issue();
                if (rs.failed) break;
            }
            const int slot = rs.taken % kDepth;
            if (!__all_sync(0xffffffffu, mbar_wait_bounded(&br.full[slot], uint32_t(rs.taken / kDepth) & 1,
                                                           ctl.wait_ns))) {
                rs.failed = true;
                break;
            }
            const SlotHdr h = br.hdr[slot];
            const int nu = (h.count + UNIT - 1) / UNIT;
            const int q0 = nu * warp / WARPS, q1 = nu * (warp + 1) / WARPS, nq = q1 - q0;
            const double4* share = sm.ring + slot * kTile + q0 * UNIT;
            const int ns = min(h.count, q1 * UNIT) - q0 * UNIT;
            bool space = nq > 0 && !flat;
            if (nq > 0 && flat) {
                Plane plane;
                plane.load(*ps);
                space = !map_share<PSI, SHARE>(share, mapped, ns, plane, wsum, lsum);
            }
            if (space) {
                const double4* tgt = src + t0 + c0;
                int g = 0;
                for (; g + 2 <= full; g += 2)
                    space_fold<PSI, 2>(share, 0, ns, 1, tgt + 32 * g + lane, acc3 + 32 * g,
                                       PSI ? accp + 32 * g : accp, sm.lg);
                if (g < full)
                    space_fold<PSI, 1>(share, 0, ns, 1, tgt + 32 * g + lane, acc3 + 32 * g,
                                       PSI ? accp + 32 * g : accp, sm.lg);
                if (r > 0)
                    space_fold<PSI, 1>(share, lane % L, ns, L, tgt + 32 * full + min(lane / L, r - 1),
                                       acc3 + 32 * full, PSI ? accp + 32 * full : accp, sm.lg);
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&br.empty[slot]);
            rs.taken++;
            if (h.count == 0) break;
            if (nq > 0 && !space) {
                const bool gd = h.guard != 0;
                const auto* tp = sm.tpos + lane;
                switch (full) {
                    case 1: plane_fold<PSI, SHARE, 1>(mapped, 0, nq, 1, gd, tp, acc, accp, wz, sm.lg); break;
                    case 2: plane_fold<PSI, SHARE, 2>(mapped, 0, nq, 1, gd, tp, acc, accp, wz, sm.lg); break;
                    case 3: plane_fold<PSI, SHARE, 3>(mapped, 0, nq, 1, gd, tp, acc, accp, wz, sm.lg); break;
                    case 4: plane_fold<PSI, SHARE, 4>(mapped, 0, nq, 1, gd, tp, acc, accp, wz, sm.lg); break;
                }
                if (r > 0)
                    plane_fold<PSI, SHARE, 1>(mapped, lane % L, nq, L, gd, sm.tpos + 32 * full + min(lane / L, r - 1),
                                                acc + 32 * full, PSI ? accp + 32 * full : accp, wz + 32 * full,
                                             sm.lg);
                __syncwarp();  // the share is used up before the next one is mapped over it
            }
        }
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            wsum += __shfl_xor_sync(0xffffffffu, wsum, off);
            if (PSI) lsum += __shfl_xor_sync(0xffffffffu, lsum, off);
        }
        if (lane == 0) {
            sm.wsum[warp] = wsum;
            sm.lsum[warp] = lsum;
        }
        if (warp > 0) rs.issued = rs.taken;
        // every tile issued for this chunk has been taken, so the counters
        // agree in every warp unless a wait gave up
        rs.failed = __syncthreads_or(rs.failed) != 0;
        if (rs.failed) {
            // no bulk copy may still be landing in this block's shared memory
            // when it exits: warp 0 waits (bounded) for the tiles not known to
            // have landed -- at most the last kDepth it issued
            if (warp == 0)
                for (int t = max(0, max(rs.issued - kDepth, rs.taken)); t < rs.issued; t++)
                    mbar_wait_bounded(&br.full[t % kDepth], uint32_t(t / kDepth) & 1, ctl.wait_ns);
            return;
        }
        // the targets' sums over the warps (and lanes)
        for (int tgt = tid; tgt < cn; tgt += 32 * WARPS) {
            const double4 v = src[t0 + c0 + tgt];
            const double x = v.x, y = v.y, z = v.z;
            const bool rest = tgt >= 32 * full;
            const int s0 = rest ? 32 * full + L * (tgt - 32 * full) : tgt, ns = rest ? L : 1;
            double bu = 0, bv = 0, bp = 0, bz = 0, wtot = 0, ltot = 0;
            Acc3 in_space{};
            for (int w = 0; w < WARPS; w++) {
                wtot += sm.wsum[w];
                ltot += sm.lsum[w];
                for (int k = s0; k < s0 + ns; k++) {
                    const Acc& a = sm.acc[w * kSlots + k];
                    bu += a.u;
                    bv += a.v;
                    const Acc3& a3 = sm.acc3[w * kSlots + k];
                    in_space.x += a3.x;
                    in_space.y += a3.y;
                    in_space.z += a3.z;
                    bz += sm.wz[w * kSlots + k];
                    if (PSI) bp += sm.accp[w * kSlots + k];
                }
            }
            double4 o = make_double4(0.0, 0.0, 0.0, bp);
            if (flat) {
                const double2 p = sm.tpos[tgt];
                o = target_sum<PSI>(*ps, wtot, ltot, x, y, z, p.x, p.y, bu, bv, bp, bz);
            }
            o.x += in_space.x;
            o.y += in_space.y;
            o.z += in_space.z;
            partials[int64_t(it.part) * pstride + t0 + c0 + tgt] = o;
        }
        __syncthreads();
    }
}

__device__ __forceinline__ void init_ring(const PairBars& br, int warps, int depth) {
    if (threadIdx.x == 0) {
        for (int d = 0; d < depth; d++) {
            mbar_init(&br.full[d], 1);
            mbar_init(&br.empty[d], warps);
        }
        mbar_init_fence();
    }
    __syncthreads();
}

// Blocks per SM that the registers must allow: 128 a thread, four blocks of
// four warps (at 96 and five blocks the level-7 treecode took 0.958 ms per
// right-hand side instead of 0.939).
constexpr int blocks_per_sm(int threads) { return 65536 / 128 / threads; }

// One block per work item; a ring of kDepth tile slots.
template <int THREADS, bool PSI>
__global__ void __launch_bounds__(THREADS, blocks_per_sm(THREADS))
    k_plane_pairs(const double4* __restrict__ src, const Segment* __restrict__ segs,
                  const int32_t* __restrict__ leaf_start, const WorkItem* __restrict__ items,
                  double4* __restrict__ partials, int64_t pstride, int* __restrict__ err, const PairCtl ctl) {
    constexpr int WARPS = THREADS / 32;
    extern __shared__ __align__(128) unsigned char smem_raw[];
    __shared__ __align__(8) uint64_t full_bar[kDepth], empty_bar[kDepth];
    __shared__ SlotHdr hdr[kDepth];
    __shared__ PlaneShared plane;
    const PairBars br{full_bar, empty_bar, hdr, &plane};
    init_ring(br, WARPS, kDepth);
    RingState rs{0, 0, false};
    auto& sm = *reinterpret_cast<PairSmem<WARPS, PSI>*>(smem_raw);
    if (PSI && threadIdx.x < 32) sm.lg[threadIdx.x] = log2(1.0 + threadIdx.x / 32.0);  // read after run_item's barriers
    const WorkItem it = items[blockIdx.x];
    run_item<WARPS, PSI>(it, src, segs, leaf_start, partials, pstride,
                         sm, br, rs, ctl,
                         int(blockIdx.x) == ctl.hold_block);
    if (rs.failed && threadIdx.x == 0) set_error(err, kErrTimeout);
}

template <int THREADS, bool PSI>
static cudaError_t run_pairs(cudaStream_t st, int nitems, const void* src, const Segment* segs,
                             const int32_t* leaf_start, const WorkItem* items, double4* partials, int64_t pstride,
                             int* err, PairCtl ctl) {
    constexpr size_t smem = sizeof(PairSmem<THREADS / 32, PSI>);
    const cudaError_t e = allow_smem(k_plane_pairs<THREADS, PSI>, smem);
    if (e != cudaSuccess) return e;
    k_plane_pairs<THREADS, PSI><<<nitems, THREADS, smem, st>>>(static_cast<const double4*>(src), segs, leaf_start,
                                                               items, partials, pstride, err, ctl);
    return cudaGetLastError();
}

template <bool PSI>
static cudaError_t dispatch(cudaStream_t st, int warps, int nitems, const void* src, const Segment* segs,
                            const int32_t* leaf_start, const WorkItem* items, double4* partials, int64_t pstride,
                            int* err, PairCtl ctl) {
    switch (warps) {
        case 4: return run_pairs<128, PSI>(st, nitems, src, segs, leaf_start, items, partials, pstride, err, ctl);
        case 5: return run_pairs<160, PSI>(st, nitems, src, segs, leaf_start, items, partials, pstride, err, ctl);
        case 6: return run_pairs<192, PSI>(st, nitems, src, segs, leaf_start, items, partials, pstride, err, ctl);
        case 8: return run_pairs<256, PSI>(st, nitems, src, segs, leaf_start, items, partials, pstride, err, ctl);
    }
    return cudaErrorInvalidConfiguration;
}

cudaError_t launch_plane_pairs(cudaStream_t st, bool psi, int warps, int nitems, const void* src, const Segment* segs,
                               const int32_t* leaf_start, const WorkItem* items, double4* partials, int64_t pstride,
                               int* err, PairCtl ctl) {
    if (nitems == 0) return cudaSuccess;
    return psi ? dispatch<true>(st, warps, nitems, src, segs, leaf_start, items, partials, pstride, err, ctl)
               : dispatch<false>(st, warps, nitems, src, segs, leaf_start, items, partials, pstride, err, ctl);
}

}  // namespace fss
