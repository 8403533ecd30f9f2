"""The dual tree's starting nodes (Tree::loadBalancedBreak) where sizes tie: on lattices and duplicated bodies most
nodes of a level hold equally many, and which of them is split follows the host's heap. The interaction
counts depend on the starting nodes, so they must equal the oracle's; clustered sets take the counting form."""
import numpy as np
import pytest

from test_gpu_dual import dual_solver, two_spheres

pytestmark = pytest.mark.gpu


def check_counts(nb, oracle, pm, leaf, theta):
    _, ref = oracle.dual_accelerations(pm, G=1.0, eps=1e-4, theta=theta, leaf=leaf)
    with dual_solver(nb, pm, leaf, theta) as s:
        s.update_accelerations()
        c = s.counts()
    got = [c["particle_particle"], c["node_particle"], c["particle_node"], c["node_node"]]
    assert got == [int(x) for x in ref]


@pytest.mark.parametrize("side,leaf", [(8, 64), (10, 16), (12, 4), (16, 8), (17, 2)])
def test_lattices(nb, oracle, side, leaf):
    g = np.stack(np.meshgrid(*[np.arange(side)] * 3, indexing="ij"), -1).reshape(-1, 3)
    pm = np.ones((len(g), 4), np.float32)
    pm[:, :3] = g / side
    pm[:, 3] = 1.0 / len(g)
    check_counts(nb, oracle, pm, leaf, 0.5)


@pytest.mark.parametrize("n,leaf", [(200, 1), (300, 64), (3000, 1), (20000, 16)])
def test_clustered(nb, oracle, n, leaf):
    pm, _ = two_spheres(nb, n, seed=n)
    pm[: n // 8] = pm[n // 8: 2 * (n // 8)]  # pairs of coincident bodies
    check_counts(nb, oracle, pm, leaf, 0.5)


@pytest.mark.parametrize("n,leaf", [(131_071, 32), (131_072, 32), (131_072, 16), (160_001, 8)])
def test_frontier_sizes(nb, oracle, n, leaf):
    """Both sides of the line at which the frontier and the near-field units grow, and small leaves above it."""
    pm, _ = two_spheres(nb, n, seed=4)
    check_counts(nb, oracle, pm, leaf, 0.7)
