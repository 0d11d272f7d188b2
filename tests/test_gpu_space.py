"""The FP64 sums where the plane does not serve: they must come out as sums in
space, target by target.

Bound.  A term's differences, square, reciprocal and products are 16 roundings
at most, on either side of the comparison in FP64; n terms are added in some
order (n roundings of the partial sums); the cross product and the sums' last
steps add 16 more: an error of at most (n + 32) u times the sum of the terms'
magnitudes, u = 2^-53, and the reference, summed in extended precision, adds
nothing to it.  A logarithm's terms are taken with 30 added to their magnitude:
the parts that it is put together from (log2 of distances in the plane and of
1 + rho, at most 2 + 2 log2(4 n) here) are larger than itself.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def points(n, seed):
    rng = np.random.default_rng(seed)
    s = np.zeros((n, 5))
    s[:, :3] = rng.standard_normal((n, 3))
    s[:, :3] /= np.linalg.norm(s[:, :3], axis=1, keepdims=True)
    s[:, 3] = rng.standard_normal(n) * 5
    return s, np.full(n, 4 * np.pi / n)


def in_space(s, a):
    """u, psi in extended precision, and the sums of the magnitudes of their terms."""
    x = s[:, :3].astype(np.longdouble)
    w = (s[:, 3] * a).astype(np.longdouble)
    u, psi, mu, mp = np.empty(x.shape), np.empty(len(x)), np.empty(len(x)), np.empty(len(x))
    for i in range(len(x)):
        d = x - x[i]
        r2 = (d * d).sum(1)
        other = r2 > 0
        r2 = np.where(other, r2, 1)
        f = np.where(other, w / r2, 0)
        lg = np.where(other, np.log(r2 / 2), 0)
        u[i] = -np.cross(x[i], f @ d) / (2 * np.pi)
        psi[i] = -(w @ lg) / (4 * np.pi)
        radius = np.sqrt((x[i] ** 2).sum())
        mu[i] = radius * (np.abs(f) * np.sqrt(r2)).sum() / (2 * np.pi)
        mp[i] = np.abs(w) @ (np.abs(lg) + 30) / (4 * np.pi)
    return u, psi, mu, mp


def check(fss, s, a, method, levels, built=None):
    u, psi, mu, mp = in_space(s, a)
    with fss.Context(method=method, precision=fss.PREC_FP64, tree_levels=levels, theta=1e-3) as c:
        c.set_particles(s if built is None else built, a)
        out, p = c.rhs(s, a, psi=True)
        alone = c.rhs(s, a)
    eps = (len(s) + 32) * 2.0 ** -53
    assert np.all(np.linalg.norm(out[:, :3] - u, axis=1) <= eps * mu)
    assert np.all(np.linalg.norm(alone[:, :3] - u, axis=1) <= eps * mu)
    assert np.all(np.abs(p - psi) <= eps * mp)


ALL_PAIRS = [(0, 0), (1, 1), (1, 2)]  # direct sum; trees that resolve every pair


@pytest.mark.parametrize("method,levels", ALL_PAIRS)
@pytest.mark.parametrize("radius", [0.5, 1.0, 1 + 1e-9, 1.01, 1.5, 2.0])
def test_any_radius(fss, radius, method, levels):
    s, a = points(701, 3)
    s[:, :3] *= radius
    check(fss, s, a, method, levels)


@pytest.mark.parametrize("method,levels", ALL_PAIRS)
@pytest.mark.parametrize("digits", [4, 6, 10, 14])
def test_rounded_positions(fss, digits, method, levels):
    s, a = points(660, 5)
    s[:, :3] = np.round(s[:, :3], digits)
    check(fss, s, a, method, levels)


@pytest.mark.parametrize("method,levels", ALL_PAIRS)
def test_a_few_off_the_sphere(fss, method, levels):
    """Sources and targets off the sphere among others on it."""
    s, a = points(900, 7)
    s[[3, 120, 121, 500, 899], :3] *= np.array([0.9, 1.1, 1 + 1e-12, 1.3, 1 - 1e-5])[:, None]
    check(fss, s, a, method, levels)


@pytest.mark.parametrize("method,levels", ALL_PAIRS + [(1, 3)])
@pytest.mark.parametrize("h", [1e-2, 1e-3, 1e-4, 1e-6, 1e-8])
def test_close_pairs(fss, h, method, levels):
    """Pairs h apart, of opposite weights, wherever in their leaf they lie."""
    s, a = points(1200, 9)
    near = s[:600, :3] + h * np.random.default_rng(2).standard_normal((600, 3))
    s[600:, :3] = near / np.linalg.norm(near, axis=1, keepdims=True)
    s[600:, 3] = -s[:600, 3]
    check(fss, s, a, method, levels)


@pytest.mark.parametrize("n", [1, 2, 3, 31, 33, 64, 127, 129, 160, 161, 300])
def test_one_region(fss, n):
    """Particles of a region that one plane serves, among others far away: every
    count of near and far sources in a warp's share."""
    s, a = points(n + 500, n)
    s[:n, :3] = np.array([1.0, 0.5, 0.2]) + 0.1 * s[:n, :3]
    s[:n, :3] /= np.linalg.norm(s[:n, :3], axis=1, keepdims=True)
    check(fss, s, a, 0, 0)
    check(fss, s, a, 1, 2)


def pair_time(ctx, s, a):
    """Least device time of the pair sums of one right-hand side, of 8."""
    times = []
    for _ in range(8):
        ctx.profile(True)
        ctx.rhs(s, a)
        times.append(ctx.profile_read()["pairs_fp64"][0])
    return min(times)


def test_a_tree_at_other_positions_takes_one_pass(fss):
    """Leaves whose particles lie all over the sphere cost what a sum in space
    costs (14 operations a pair for 10), not a pass over the sources for each
    group of them, which takes three times a tree's own positions and more.
    Twice is between the two."""
    s, a = points(40962, 11)
    t = s.copy()
    t[:, :3] = s[np.random.default_rng(1).permutation(len(s)), :3]
    with fss.Context(precision=fss.PREC_FP64) as c:
        c.set_particles(s, a)
        assert pair_time(c, t, a) < 2 * pair_time(c, s, a)


@pytest.mark.parametrize("n", [15000, 15001])
def test_direct_order_only_where_it_pays(fss, n):
    """Up to 15,000 particles the direct sum keeps the caller's order (the
    spatial one takes eight launches a step, which cost 6,000 particles a third
    more); beyond, the sums come out the same from the spatial order."""
    s, a = points(n, 13)
    x, w = s[:, :3].astype(np.longdouble), (s[:, 3] * a).astype(np.longdouble)
    with fss.Context(method=fss.METHOD_DIRECT, precision=fss.PREC_FP64) as c:
        c.set_particles(s, a)
        out = c.rhs(s, a)
        c.profile(True)
        c.rk4_step(0.01)
        assert ("order" in c.profile_read()) == (n > 15000)
    for i in (0, 1, n // 2, n - 2, n - 1):
        d = x - x[i]
        r2 = (d * d).sum(1)
        r2[i] = 1
        f = w / r2
        u = -np.cross(x[i], f @ d) / (2 * np.pi)
        assert np.linalg.norm(out[i, :3] - u) <= (n + 32) * 2.0 ** -53 * (np.abs(f) * np.sqrt(r2)).sum() / (2 * np.pi)


def test_ordered_direct_steps_resume_bit_for_bit(fss):
    s, a = points(15600, 17)
    with fss.Context(method=fss.METHOD_DIRECT, precision=fss.PREC_FP64) as c:
        c.set_particles(s, a)
        c.rk4_step(0.01)
        mid = c.get_state()
        c.rk4_step(0.01)
        end = c.get_state()
    with fss.Context(method=fss.METHOD_DIRECT, precision=fss.PREC_FP64) as c:
        c.set_particles(mid, a)
        c.rk4_step(0.01)
        assert np.array_equal(c.get_state(), end)
