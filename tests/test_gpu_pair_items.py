"""The FP32 pair engine: how its work is laid out (warps of a block, targets of
an item, chunks of a leaf) must not show in the result, bit for bit, and leaves
of every remainder must come out right."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def spread(n, seed):
    rng = np.random.default_rng(seed)
    s = np.zeros((n, 5))
    s[:, :3] = rng.standard_normal((n, 3))
    s[:, :3] /= np.linalg.norm(s[:, :3], axis=1, keepdims=True)
    s[:, 3] = rng.standard_normal(n) * 5
    return s, np.full(n, 4 * np.pi / n)


def in_space(s, a, rows=slice(None)):
    """(u, psi, and the sums of the magnitudes of their terms) at FP32 positions and weights, in FP64."""
    x, w = s[:, :3], (s[:, 3] * a).astype(np.float32).astype(float)
    d = x[None, :, :] - x[rows, None, :]
    r2 = np.sum(d * d, axis=2)
    same = r2 == 0
    r2[same] = 1.0
    f = w[None, :] / r2
    f[same] = 0.0
    u = -np.cross(x[rows], np.einsum("ij,ijk->ik", f, d)) / (2 * np.pi)
    lg = np.log(r2 / 2)
    lg[same] = 0.0
    return (u, -lg @ w / (4 * np.pi), np.sum(np.abs(f) * np.sqrt(r2), axis=1) / (2 * np.pi),
            (np.abs(lg) + 1) @ np.abs(w) / (4 * np.pi))


# one leaf per face: leaves of about 1, 5, 16, 32, 48, 100, 160, 165 targets
@pytest.mark.parametrize("n", [20, 100, 320, 640, 960, 2000, 3200, 3300])
@pytest.mark.parametrize("method", [0, 1])
def test_every_remainder(fss, n, method):
    """A tile's sum adds 128 terms, of 6 roundings each, on a lane: within 134
    half-units in the last place (8e-6) of the sum of their magnitudes; one
    missing or repeated source is a 1/n-th of it."""
    s, a = spread(n, n)
    s[:, :3] = s[:, :3].astype(np.float32)
    u, psi, mu, mp = in_space(s, a)
    with fss.Context(method=method, precision=fss.PREC_MIXED, tree_levels=1, theta=1e-3) as c:
        c.set_particles(s, a)
        out, p = c.rhs(s, a, psi=True)
    assert np.all(np.linalg.norm(out[:, :3] - u, axis=1) <= 8e-6 * mu)
    assert np.all(np.abs(p - psi) <= 8e-6 * mp)


@pytest.mark.parametrize("n,levels,clusters", [(700, 1, 0), (5001, 2, 0), (20011, 3, 1), (40000, 3, 0)])
def test_layout_does_not_show(fss, n, levels, clusters):
    s, a = spread(n, n + 1)
    kw = dict(tree_levels=levels, src_parts=2, cluster_targets=clusters)
    outs = []
    for block in (0, 160, 192, 224, 288):
        with fss.Context(block_threads=block, **kw) as c:
            c.set_particles(s, a)
            c.rk4_step(0.01, nsteps=2)
            outs.append((c.get_state(), *c.rhs(s, a, psi=True)))
    for o in outs[1:]:
        assert all(np.array_equal(x, y) for x, y in zip(o, outs[0]))


def test_direct_blocks_do_not_show(fss):
    s, a = spread(3001, 3)
    outs = []
    for block in (160, 192, 224, 288):
        with fss.Context(method=fss.METHOD_DIRECT, src_parts=3, block_threads=block) as c:
            c.set_particles(s, a)
            outs.append(c.rhs(s, a))
    # 32-target groups start at multiples of the block's targets: the last group's remainder is the same
    assert all(np.array_equal(o, outs[0]) for o in outs[1:])


def test_direct_uneven_items(fss):
    """Targets in items of 256, 128 and 64, every kind and its last rows (the bound of test_every_remainder)."""
    n = 12001
    s, a = spread(n, n)
    s[:, :3] = s[:, :3].astype(np.float32)
    rows = np.concatenate([np.arange(0, n, 97), np.arange(n - 70, n)])
    u, psi, mu, mp = in_space(s, a, rows)
    with fss.Context(method=fss.METHOD_DIRECT, precision=fss.PREC_MIXED) as c:
        c.set_particles(s, a)
        out, p = c.rhs(s, a, psi=True)
    assert np.all(np.linalg.norm(out[rows, :3] - u, axis=1) <= 8e-6 * mu)
    assert np.all(np.abs(p[rows] - psi) <= 8e-6 * mp)


def pair_ms(ctx, psi=False):
    times = []
    for _ in range(10):
        ctx.profile(True)
        ctx.rhs_current(psi=psi)
        times.append(ctx.profile_read()["pairs_mixed"][0])
    return min(times)


@pytest.mark.parametrize("clusters", [0, 1])
def test_stream_function_costs_its_logarithm(fss, clusters):
    """A logarithm a pair makes the sums 1.3 times as long (two operations of the
    pipe that the reciprocal needs instead of one); with its loop unrolled eight
    times it was 1.6 to 1.7 times."""
    s, a = spread(163842, 3)
    with fss.Context(cluster_targets=clusters) as c:
        c.set_particles(s, a)
        assert pair_ms(c, True) < 1.47 * pair_ms(c)


def test_direct_items_fit_one_round(fss):
    """3,700 particles in items of 32 targets would be one and a half rounds of
    blocks, and longer sums than those of 4,300; 7,000 in 64s two rounds. Each
    must stay within 4% of the line through its neighbours (14% and 7% above it
    otherwise)."""
    ms = {}
    for n in (3000, 3700, 4300, 6000, 7000, 8000):
        s, a = spread(n, n)
        with fss.Context(method=fss.METHOD_DIRECT) as c:
            c.set_particles(s, a)
            ms[n] = pair_ms(c)
    assert ms[3700] < 1.04 * (ms[3000] + (ms[4300] - ms[3000]) * 700 / 1300), ms
    assert ms[7000] < 1.04 * (ms[6000] + ms[8000]) / 2, ms


@pytest.mark.parametrize("block", [160, 192, 224, 288])
@pytest.mark.parametrize("clusters", [0, 1])
def test_block_threads_cost_nothing(fss, block, clusters):
    """block_threads counts in the source split only: with the split given, the
    sums take the same time (five, six and eight warps took up to 16% longer)."""
    s, a = spread(40962, 5)
    ms = []
    for b in (0, block):
        with fss.Context(block_threads=b, src_parts=4, cluster_targets=clusters) as c:
            c.set_particles(s, a)
            ms.append(pair_ms(c))
    assert ms[1] < 1.04 * ms[0]
