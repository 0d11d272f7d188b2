// k_plane.cu -- the FP64 pair engine: direct sum, near field and far field,
// summed in the plane, what is near in space.
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
// target.
//
// A difference in the plane carries the map's rounding, a few u |xi| (u =
// 2^-53), where one in space is exact for neighbours: relative to a pair h
// apart, a few u |xi| / h.  So the plane takes only sources beyond kNear times
// the targets' largest |xi|, each target at least a fifth of |xi_j| away.  And
// the map holds on the unit sphere alone and serves targets on c's side of it
// (kMinCos).  What it does not serve is summed in space, at 14 operations a
// pair: sources near the targets or off the sphere (kOnSphere), and every
// source of a direct sum in the caller's order (WorkItem::space) or for a chunk
// with a target off the sphere or with targets all over it (a tree evaluated at
// other positions than its own: 163,842 particles 1.26 ms, where a pass over the
// sources around each group of targets took 4.26).
//
// Bound by the FP64 pipe, 79% busy in the first of these.  Pair sums of one
// right-hand side, all in space by one target a lane and here: treecode of
// 163,842 particles (n = 8, theta = 0.7) 1.314 and 0.960 ms (0.925 with all
// sources but the targets in the plane), with target clusters (n = 10) 0.719 and
// 0.557; direct sum of 20,011 particles 0.402 and 0.323; 40,962 particles with the
// stream function 1.144 and 0.453.
// The FP32 engine (k_pairs.cu) sums in space.
#include <algorithm>

#include "pairs_common.cuh"

namespace fss {

constexpr int kUnroll = 2;       // units per step of the pair loop
constexpr int kDepth = 2;        // ring depth (tiles in flight)
constexpr int kTile = kTileSources;
constexpr double kMinCos = 0.2;  // the plane serves targets with x.c above this
constexpr int kSlots = 32 * (kMaxFull + 1);  // accumulator slots of a warp

// Sources with |xi| up to this times the targets' largest (and to the distance
// below which a position's rounding across the sphere would show) are near.
// Direct sums of 2,001 to 163,842 random particles, plainly summed, come out to
// 2.2e-16 to 5.2e-16 of the result with it as with 1.5, 2 and 3 (in space 8e-16
// to 1.4e-14, in longer sums); the level-7 treecode above 0.982, at 1.5 0.996 ms,
// before the rest of its targets took a lane's next place.
constexpr double kNear = 1.25;
constexpr double kNearest = 1e-6;
// What the pair loop in space adds to r^2, so that a source at the target's
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
    int flat;   // it serves them
    int reach;  // the largest |xi|^2 of them (a float rounded up, its bits)
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

// Stereographic coordinates of x / |x|, x on the sphere but for rounding: xi =
// (x.e1, x.e2) / (|x| + x.c).  With t = x - c on c's side, |x| + x.c =
// ((1 + |x|)^2 - |t|^2) / 2, and (1 + |x|)^2 = 2 + 2 |x|^2; with t = x + c on
// the other, |t|^2 / 2 (and x.e = t.e either way); close to the antipode -c,
// where t's radial part is rounding, |t|^2 = 2 (1 - sqrt(1 - q)) with q =
// (t.e1)^2 + (t.e2)^2.  Explicitly rounded operations: a target and the same
// point as a source map to the same bits, so that it is among the near.
__device__ __forceinline__ void plane_map(const Plane& p, double x, double y, double z, double& u, double& v) {
    const double nn = norm2(x, y, z);
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
    const double k = rcp_fast(far ? __dmul_rn(0.5, tt) : __fma_rn(-0.5, tt, __dadd_rn(1.0, nn)));
    u = __dmul_rn(a, k);
    v = __dmul_rn(b, k);
}
__device__ __forceinline__ double rho_of(double u, double v) { return __fma_rn(v, v, __dmul_rn(u, u)); }

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
// sums with the stream function of 40,962 particles 1.00 ms with log2(), 0.46 ms
// with this.
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
// SHARE entries, padded to whole units with w = 0), none of them near.
//
// The reciprocal is the hardware approximation y of 1 / r^2 (relative error
// e < 2^-18) refined by y (1 + e + e^2), error e^3 < 2^-54, folded into the
// product with w.
template <bool PSI, int SHARE, int NT>
__device__ __forceinline__ void plane_pairs(const double* __restrict__ s, int q0, int q1, int step,
                                            const double2 (&t)[NT], double (&bu)[NT], double (&bv)[NT],
                                            double (&ap)[NT], const double* __restrict__ lg) {
#pragma unroll
    for (int k = 0; k < NT; k++) bu[k] = bv[k] = ap[k] = 0.0;
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
                const double r2 = fma(dv, dv, du * du);
                const double y = rcp_seed(r2);
                const double e = fma(-r2, y, 1.0);
                const double wy = qw[h] * y;
                const double sc = fma(wy, fma(e, e, e), wy);
                bu[k] = fma(sc, du, bu[k]);
                bv[k] = fma(sc, dv, bv[k]);
                if (PSI) ap[k] = fma(qw[h], log2_beside(r2, y, lg), ap[k]);
            }
    }
}

// A warp's share of a tile for its lanes' NT targets (positions tpos[32 k]),
// added to the lane's accumulators.
template <bool PSI, int SHARE, int NT>
__device__ __forceinline__ void plane_fold(const double* __restrict__ share, int q0, int q1, int step,
                                           const double2* tpos, Acc* acc, double* accp, const double* lg) {
    const int lane = threadIdx.x & 31;
    double2 t[NT];
    double bu[NT], bv[NT], bp[NT];
#pragma unroll
    for (int k = 0; k < NT; k++) t[k] = tpos[32 * k];
    plane_pairs<PSI, SHARE, NT>(share, q0, q1, step, t, bu, bv, bp, lg);
#pragma unroll
    for (int k = 0; k < NT; k++) {
        Acc& a = acc[32 * k + lane];
        a.u += bu[k];
        a.v += bv[k];
        if (PSI) accp[32 * k + lane] += bp[k];
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
#pragma unroll(PSI ? 2 : 4)
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

// Such sources of a warp's share of a tile for its lanes' NT targets (tgt, and
// for NT = 2 tgt1), added to the lane's accumulators.
template <bool PSI, int NT>
__device__ __forceinline__ void space_fold(const double4* __restrict__ share, int j0, int n, int step,
                                           const double4* __restrict__ tgt, const double4* __restrict__ tgt1,
                                           Acc3* acc, double* accp,
                                           const double* lg) {
    const int lane = threadIdx.x & 31;
    double4 t[NT];
    Acc3 a[NT];
    double ap[NT];
#pragma unroll
    for (int k = 0; k < NT; k++) t[k] = k == 0 ? *tgt : *tgt1;
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

// A warp's share of a landed tile -- n sources, `in` -- parted: those that the
// plane serves are mapped to it, into the warp's own arrays u, v, w of SHARE
// entries, padded to whole units with w = 0 (nf of them, their sums of w and w
// log2(1 + rho) added to wsum and lsum); those off the sphere or near the
// targets (|xi|^2 <= near2) move to the front of `in` (nn of them).
template <bool PSI, int SHARE>
__device__ __forceinline__ void part_share(double4* __restrict__ in, double* __restrict__ out, int n, const Plane& p,
                                           double near2, int& nf, int& nn, double& wsum, double& lsum) {
    constexpr int ROUNDS = (SHARE + 31) / 32;
    const int lane = threadIdx.x & 31;
    const unsigned below = (1u << lane) - 1;
    double4 q[ROUNDS];
#pragma unroll
    for (int i = 0; i < ROUNDS; i++)
        if (32 * i + lane < n) q[i] = in[32 * i + lane];
    __syncwarp();  // all read before any is overwritten
    nf = nn = 0;
#pragma unroll
    for (int i = 0; i < ROUNDS; i++) {
        const bool any = 32 * i + lane < n;
        double u = 0, v = 0;
        bool far = false;
        if (any) {
            plane_map(p, q[i].x, q[i].y, q[i].z, u, v);
            far = on_sphere(q[i].x, q[i].y, q[i].z) && rho_of(u, v) > near2;
        }
        const unsigned fars = __ballot_sync(0xffffffffu, far), nears = __ballot_sync(0xffffffffu, any && !far);
        if (far) {
            const int k = nf + __popc(fars & below);
            out[k] = u;
            out[SHARE + k] = v;
            out[2 * SHARE + k] = q[i].w;
            wsum += q[i].w;
            if (PSI) lsum += q[i].w * lg2_fast(fma(v, v, fma(u, u, 1.0)));
        } else if (any) {
            in[nn + __popc(nears & below)] = q[i];
        }
        nf += __popc(fars);
        nn += __popc(nears);
    }
    if (lane == 0 && (nf & 1)) {
        out[nf] = kFarAway;
        out[SHARE + nf] = 0.0;
        out[2 * SHARE + nf] = 0.0;
    }
    if (nn > 0) fence_proxy_async_smem();  // before the slot's next copy lands over them
}

// Tile header (sources) written by warp 0 before the slot's arrive (every warp
// reads it after the slot's phase completes).
struct SlotHdr {
    int count;
};

struct RingState {
    int issued, taken;  // tiles, over all chunks
    bool failed;
};

// A target's A (and its log2 sum) from the sums in the plane.
template <bool PSI>
__device__ __forceinline__ double4 target_sum(const PlaneShared& ps, double wtot, double ltot, double x, double y, double z, double tu, double tv,
                                              double bu, double bv, double bp) {
    const double u = tu, v = tv, rho = u * u + v * v;
    const double W = wtot, f = W / (1.0 + rho);
    const double p1 = bu + f * u, p2 = bv + f * v;
    const double g = 0.5 * (1.0 + rho), h = p1 * u + p2 * v;
    const double k1 = g * p1 - h * u, k2 = g * p2 - h * v, kx = 0.5 * W;
    double4 o;
    o.x = k1 * ps.e1[0] + k2 * ps.e2[0] - h * ps.c[0] - kx * x;
    o.y = k1 * ps.e1[1] + k2 * ps.e2[1] - h * ps.c[1] - kx * y;
    o.z = k1 * ps.e1[2] + k2 * ps.e2[2] - h * ps.c[2] - kx * z;
    o.w = 0.0;
    if (PSI)  // log2 |x_j - x_i|^2 = log2 |xi_j - xi_i|^2 + 2 - log2(1 + rho_i) - log2(1 + rho_j)
        o.w = bp + W * (2.0 - log2(1.0 + rho)) - ltot;
    return o;
}

// Shared memory of a pair block: the landing ring (kDepth tiles as copied),
// and each warp's parted share of a tile, accumulators and sums over its
// sources; the targets' plane coordinates.
template <int WARPS, bool PSI>
struct PairSmem {
    static constexpr int kShare = (kTile / 2 + WARPS - 1) / WARPS * 2;
    double4 ring[kDepth * kTile];
    double mapped[WARPS * 3 * kShare];
    Acc acc[WARPS * kSlots];
    Acc3 acc3[WARPS * kSlots];
    double2 tpos[kSlots];
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
// parts its share of a landed tile, sums those in space from the slot, releases
// it through empty, and sums those in the plane, each for all targets of the
// chunk: cn >> 5 targets a lane (a source loaded serves them all) and, for the
// r = cn & 31 left over, L = 32 / r lanes a target, which split the share
// between them, or one more target a lane where L is 1 anyway.  So the
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
        const int merge = (cn & 31) > 16 && (cn >> 5) < kMaxFull ? 1 : 0;  // the rest as one more a lane
        const int full = (cn >> 5) + merge, r = merge ? 0 : cn & 31;
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
                bool with_targets;  // (near shares need no telling)
                cnt = pack_tile<double4, kTile, true>(segs, leaf_start, it.g1, win, t0, t0 + nt, src,
                                                      sm.ring + slot * kTile, &br.full[slot], with_targets);
                if (lane == 0) {
                    br.hdr[slot].count = cnt;
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
            for (int i = lane; i < cn && !it.space; i += 32) {
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
                ps->flat = !it.space;
                ps->reach = 0;
            }
        }
        Acc* acc = sm.acc + warp * kSlots;
        Acc3* acc3 = sm.acc3 + warp * kSlots;
        double* accp = PSI ? sm.accp + warp * kSlots : sm.accp;
        double* mapped = sm.mapped + warp * 3 * SHARE;
        for (int k = lane; k < 32 * (full + 1); k += 32) {
            acc[k] = Acc{};
            acc3[k] = Acc3{};
            if (PSI) accp[k] = 0.0;
        }
        __syncthreads();
        if (!it.space) {
            Plane plane;
            plane.load(*ps);
            for (int i = tid; i < max(cn, 32 * full); i += 32 * WARPS) {
                const double4 v = src[t0 + c0 + min(i, cn - 1)];
                double2 p;
                plane_map(plane, v.x, v.y, v.z, p.x, p.y);
                sm.tpos[i] = p;
                if (on_sphere(v.x, v.y, v.z) && plane.serves(v.x, v.y, v.z))
                    atomicMax(&ps->reach, __float_as_int(__double2float_ru(rho_of(p.x, p.y))));
                else
                    ps->flat = 0;
            }
        }
        __syncthreads();
        const bool flat = ps->flat != 0;
        const double near2 = fmax(kNear * kNear * double(__int_as_float(ps->reach)), kNearest * kNearest);
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
            double4* share = sm.ring + slot * kTile + q0 * UNIT;
            const int ns = min(h.count, q1 * UNIT) - q0 * UNIT;
            int nf = 0, nn = 0;
            if (flat) {
                Plane plane;
                plane.load(*ps);
                part_share<PSI, SHARE>(share, mapped, ns, plane, near2, nf, nn, wsum, lsum);
            } else if (nq > 0) {
                nn = ns;
            }
            __syncwarp();
            if (nn > 0) {
                const double4* tgt = src + t0 + c0;
                int g = 0;
                for (; g + 2 <= full; g += 2)
                    space_fold<PSI, 2>(share, 0, nn, 1, tgt + 32 * g + lane, tgt + min(32 * g + 32 + lane, cn - 1),
                                       acc3 + 32 * g, PSI ? accp + 32 * g : accp, sm.lg);
                if (g < full)
                    space_fold<PSI, 1>(share, 0, nn, 1, tgt + min(32 * g + lane, cn - 1), nullptr, acc3 + 32 * g,
                                       PSI ? accp + 32 * g : accp, sm.lg);
                if (r > 0)
                    space_fold<PSI, 1>(share, lane % L, nn, L, tgt + 32 * full + min(lane / L, r - 1), nullptr,
                                       acc3 + 32 * full, PSI ? accp + 32 * full : accp, sm.lg);
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&br.empty[slot]);
            rs.taken++;
            if (h.count == 0) break;
            if (nf > 0) {
                const int nu = (nf + UNIT - 1) / UNIT;
                const auto* tp = sm.tpos + lane;
                switch (full) {
                    case 1: plane_fold<PSI, SHARE, 1>(mapped, 0, nu, 1, tp, acc, accp, sm.lg); break;
                    case 2: plane_fold<PSI, SHARE, 2>(mapped, 0, nu, 1, tp, acc, accp, sm.lg); break;
                    case 3: plane_fold<PSI, SHARE, 3>(mapped, 0, nu, 1, tp, acc, accp, sm.lg); break;
                    case 4: plane_fold<PSI, SHARE, 4>(mapped, 0, nu, 1, tp, acc, accp, sm.lg); break;
                }
                if (r > 0)
                    plane_fold<PSI, SHARE, 1>(mapped, lane % L, nu, L, sm.tpos + 32 * full + min(lane / L, r - 1),
                                              acc + 32 * full, PSI ? accp + 32 * full : accp, sm.lg);
            }
            __syncwarp();  // the share is used up before the next one takes its place
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
        if (r > 0 && L > 1) {  // the lanes of a target left over: their sums to the first of them
            Acc& a = acc[32 * full + lane];
            Acc3& a3 = acc3[32 * full + lane];
            const int sub = lane % L;
            a.u = group_sum(a.u, sub, L);
            a.v = group_sum(a.v, sub, L);
            a3.x = group_sum(a3.x, sub, L);
            a3.y = group_sum(a3.y, sub, L);
            a3.z = group_sum(a3.z, sub, L);
            if (PSI) accp[32 * full + lane] = group_sum(accp[32 * full + lane], sub, L);
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
        // the targets' sums over the warps
        for (int tgt = tid; tgt < cn; tgt += 32 * WARPS) {
            const double4 v = src[t0 + c0 + tgt];
            const double x = v.x, y = v.y, z = v.z;
            const int k = tgt >= 32 * full ? 32 * full + L * (tgt - 32 * full) : tgt;
            double bu = 0, bv = 0, bp = 0, wtot = 0, ltot = 0;
            Acc3 in_space{};
            for (int w = 0; w < WARPS; w++) {
                wtot += sm.wsum[w];
                ltot += sm.lsum[w];
                const Acc& a = sm.acc[w * kSlots + k];
                bu += a.u;
                bv += a.v;
                const Acc3& a3 = sm.acc3[w * kSlots + k];
                in_space.x += a3.x;
                in_space.y += a3.y;
                in_space.z += a3.z;
                if (PSI) bp += sm.accp[w * kSlots + k];
            }
            double4 o = make_double4(0.0, 0.0, 0.0, bp);
            if (flat) {
                const double2 p = sm.tpos[tgt];
                o = target_sum<PSI>(*ps, wtot, ltot, x, y, z, p.x, p.y, bu, bv, bp);
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
// four warps, as many as the shared memory holds.
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

cudaError_t launch_plane_pairs(cudaStream_t st, bool psi, int nitems, const void* src, const Segment* segs,
                               const int32_t* leaf_start, const WorkItem* items, double4* partials, int64_t pstride,
                               int* err, PairCtl ctl) {
    if (nitems == 0) return cudaSuccess;
    auto run = psi ? run_pairs<128, true> : run_pairs<128, false>;
    return run(st, nitems, src, segs, leaf_start, items, partials, pstride, err, ctl);
}

}  // namespace fss
