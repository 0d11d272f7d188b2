"""The batched V^-1 products of the upward and downward passes in blocks of 4, 8
and 16 tasks, and the evaluation of leaves below and above 128 particles,
against the FP64 direct sum."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def field(fss, oracle):
    s, a = fss.make_state(6, "rh_vortices", n_vortex=8, seed=3)
    return s, a, oracle.rhs_direct(s, a)


# tree_levels 2 to 5 at 40,962 particles: leaves of 512, 128, 32 and 8, and
# about 100, 420, 1700 and 6800 clusters
@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("levels,degree", [(2, 5), (3, 6), (3, 11), (4, 5), (4, 8), (5, 6), (5, 7)])
def test_task_blocks(fss, field, prec, levels, degree):
    """Bound: interpolation in a well-separated face at theta = 0.7 converges
    as (theta / (1 + sqrt(1 - theta^2)))^(n + 1) = 0.408^(n + 1); a product
    read from a wrong task or row is wrong at O(1)."""
    s, a, ref = field
    with fss.Context(method=fss.METHOD_TREECODE, precision=prec, cluster_targets=1, degree=degree, theta=0.7,
                     tree_levels=levels) as ctx:
        ctx.set_particles(s, a)
        out = ctx.rhs(s, a)
    err = np.linalg.norm(out[:, :3] - ref[:, :3]) / np.linalg.norm(ref[:, :3])
    assert err < 0.408 ** (degree + 1), err
