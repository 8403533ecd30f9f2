"""The traversal's two forms give the same bits.

Passes over few 32-target groups run a team of warps per group, larger ones one warp per group. A body set
alone takes the first form; in a batch beside a large instance it takes the second. Accelerations and
interaction counts must be equal bit for bit, at group and leaf-list remainders, for both orders,
with and without softening, and for both slab sizes.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 3, 31, 33, 500, 2049, 9000])
@pytest.mark.parametrize("order,leaf,eps,slab", [(1, 1, 1e-4, 64), (1, 64, 0.0, 64), (2, 8, 0.0, 32), (2, 16, 1e-4, 64),
                                                 (2, 64, 1e-5, 32)])
def test_team_and_single_warp_forms_agree(nb, n, order, leaf, eps, slab):
    pm, _ = nb.scenarios.plummer(max(n, 8), seed=n)
    pm = pm[:n]
    big, _ = nb.scenarios.uniform_ball(300_000, seed=7)
    cls = nb.LinearBVHSolver if order == 1 else nb.QuadrupoleLinearBVHSolver
    kw = dict(theta=0.6, max_leaf_size=leaf)
    with cls(pm, nb.Gravity(1.0, eps), **kw) as s:
        s.traversal_shape = (256, slab)
        alone, counts = s.update_accelerations(), s.counts()
    with cls(None, nb.Gravity(1.0, eps), **kw) as s:
        s.traversal_shape = (256, slab)
        s.set_instances([n, len(big)], np.concatenate([pm, big]))
        batch = s.update_accelerations()
        per = s.instance_counts()
    assert np.array_equal(alone, batch[:n])
    assert (counts["particle_particle"], counts["node_particle"]) == tuple(int(x) for x in per[0])


@pytest.mark.parametrize("n,order,leaf,eps,slab,theta", [
    (40_001, 2, 8, 1e-4, 64, 0.5),  # sizes near the largest that run teams: full rings, a walker that waits
    (60_007, 2, 16, 0.0, 64, 0.5),
    (60_007, 1, 16, 1e-4, 32, 0.3),
    (100_003, 2, 64, 0.0, 32, 0.5),
    (100_003, 1, 64, 1e-5, 64, 0.3),
])
def test_forms_agree_in_full_rings(nb, n, order, leaf, eps, slab, theta):
    pm, _ = nb.scenarios.plummer(n, seed=n)
    big, _ = nb.scenarios.uniform_ball(300_000, seed=7)
    cls = nb.LinearBVHSolver if order == 1 else nb.QuadrupoleLinearBVHSolver
    kw = dict(theta=theta, max_leaf_size=leaf)
    with cls(pm, nb.Gravity(1.0, eps), **kw) as s:
        s.traversal_shape = (256, slab)
        alone, counts = s.update_accelerations(), s.counts()
    with cls(None, nb.Gravity(1.0, eps), **kw) as s:
        s.traversal_shape = (256, slab)
        s.set_instances([n, len(big)], np.concatenate([pm, big]))
        batch = s.update_accelerations()
        per = s.instance_counts()
    assert np.array_equal(alone, batch[:n])
    assert (counts["particle_particle"], counts["node_particle"]) == tuple(int(x) for x in per[0])
