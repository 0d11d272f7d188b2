"""The FP64 pair engine's sums in the plane at the sizes and positions where it
can go wrong, against the sums in space in numpy.

Tolerances.  The reference's own rounding and the engine's are below 1e-15 of
the sum of the terms' magnitudes, which is less than 300 times the result in
these fields: 1e-12.  Positions rounded to 6 decimals are up to 9e-7 off the
sphere; the engine takes the point of the sphere below them, the reference the
point itself, which changes a pair's term by less than 3e-6 of it and the
result by less than 1e-5 (the terms add up to about three times the result).
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def points(n, seed):
    """n points in no order, spread over the sphere, the last two antipodal to the first two."""
    rng = np.random.default_rng(seed)
    x = rng.standard_normal((n, 3))
    x /= np.linalg.norm(x, axis=1, keepdims=True)
    if n >= 8:
        x[-2:] = -x[:2]
    s = np.zeros((n, 5))
    s[:, :3] = x
    s[:, 3] = rng.standard_normal(n) * 5
    return s, np.full(n, 4 * np.pi / n)


def in_space(s, a):
    x, w = s[:, :3], s[:, 3] * a
    d = x[None, :, :] - x[:, None, :]
    r2 = np.sum(d * d, axis=2)
    with np.errstate(divide="ignore"):
        f = np.where(r2 > 0, w[None, :] / r2, 0.0)
        psi = -np.where(r2 > 0, w[None, :] * np.log(r2 / 2), 0.0).sum(1) / (4 * np.pi)
    A = np.einsum("ij,ijk->ik", f, d)
    return -np.cross(x, A) / (2 * np.pi), psi


def close(got, want, tol):
    return np.linalg.norm(got - want) <= tol * np.linalg.norm(want)


@pytest.mark.parametrize("n", [2, 3, 31, 33, 127, 128, 129, 160, 161, 255, 257, 513, 1025, 2049, 4096, 4097])
def test_direct_sizes(fss, n):
    s, a = points(n, n)
    u, psi = in_space(s, a)
    with fss.Context(method=fss.METHOD_DIRECT, precision=fss.PREC_FP64) as c:
        c.set_particles(s, a)
        out = c.rhs(s, a)
        both, p = c.rhs(s, a, psi=True)
    assert close(out[:, :3], u, 1e-12) and close(both[:, :3], u, 1e-12)
    assert close(p, psi, 1e-12)


@pytest.mark.parametrize("parts,block", [(1, 160), (3, 192), (7, 224), (1, 288)])
def test_direct_splits(fss, parts, block):
    s, a = points(1301, 5)
    u, _ = in_space(s, a)
    with fss.Context(method=fss.METHOD_DIRECT, precision=fss.PREC_FP64, src_parts=parts, block_threads=block) as c:
        c.set_particles(s, a)
        assert close(c.rhs(s, a)[:, :3], u, 1e-12)


@pytest.mark.parametrize("method,levels", [(0, 0), (1, 1), (1, 2)])
def test_coincident_particles_add_nothing_to_each_other(fss, method, levels):
    s, a = points(640, 7)
    s[[5, 200, 639], :3] = s[100, :3]
    s[17, :3] = s[400, :3]
    u, psi = in_space(s, a)
    with fss.Context(method=method, precision=fss.PREC_FP64, tree_levels=levels, theta=1e-3) as c:
        c.set_particles(s, a)
        out, p = c.rhs(s, a, psi=True)
    # the stream function leaves out the target's own weight only: log(r2 / 2) of a coincident one counts as log 1/2
    for i, same in ((5, (200, 639, 100)), (200, (5, 639, 100)), (639, (5, 200, 100)), (100, (5, 200, 639)),
                    (17, (400,)), (400, (17,))):
        psi[i] += np.log(2) / (4 * np.pi) * sum(s[j, 3] * a[j] for j in same)
    assert close(out[:, :3], u, 1e-12)
    assert close(p, psi, 1e-12)


@pytest.mark.parametrize("levels", [1, 2])
def test_tree_of_other_positions(fss, levels):
    """A tree that resolves every pair, built for one set of positions and
    evaluated at another, whose leaves' particles lie all over the sphere."""
    s, a = points(900, 11)
    t, _ = points(900, 12)
    u, psi = in_space(t, a)
    with fss.Context(precision=fss.PREC_FP64, tree_levels=levels, theta=1e-3) as c:
        c.set_particles(s, a)
        out, p = c.rhs(t, a, psi=True)
    assert close(out[:, :3], u, 1e-12)
    assert close(p, psi, 1e-12)


@pytest.mark.parametrize("method,levels", [(0, 0), (1, 1)])
def test_positions_of_few_digits(fss, method, levels):
    s, a = points(700, 13)
    s[:, :3] = np.round(s[:, :3], 6)
    s[-2:, :3] = -s[:2, :3]
    u, psi = in_space(s, a)
    with fss.Context(method=method, precision=fss.PREC_FP64, tree_levels=levels, theta=1e-3) as c:
        c.set_particles(s, a)
        out, p = c.rhs(s, a, psi=True)
    assert close(out[:, :3], u, 1e-5)
    assert close(p, psi, 1e-5)


def test_rk4_steps_resume_bit_for_bit(fss):
    """The direct sum's order depends on the positions alone: a run taken up
    from its state is the run itself."""
    s, a = points(1500, 17)
    with fss.Context(method=fss.METHOD_DIRECT, precision=fss.PREC_FP64) as c:
        c.set_particles(s, a)
        c.rk4_step(0.01, nsteps=2)
        mid = c.get_state()
        c.rk4_step(0.01, nsteps=2)
        end = c.get_state()
    with fss.Context(method=fss.METHOD_DIRECT, precision=fss.PREC_FP64) as c:
        c.set_particles(mid, a)
        c.rk4_step(0.01, nsteps=2)
        assert np.array_equal(c.get_state(), end)
