"""The tree build at the edges of its climb blocks (1024 and 4096 Karras nodes) and of its prefix scans (one kernel
up to eight 2048-position tiles, two above): every node record bit-exact against the oracle."""
import numpy as np
import pytest

from test_gpu_dual import check_dual_tree, dual_solver
from test_gpu_parity import check_tree, make_solver

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,leaf", [(1024, 1), (1025, 1), (1026, 16), (2049, 3), (4096, 17), (4097, 64), (4098, 17),
                                    (8193, 1), (16382, 16), (16383, 64), (16384, 1), (20000, 17), (40001, 2)])
@pytest.mark.parametrize("order", [1, 2])
def test_records_at_block_edges(nb, oracle, n, leaf, order):
    pm, _ = nb.scenarios.plummer(n, seed=n)
    with make_solver(nb, pm, order=order, leaf=leaf) as s:
        s.update_accelerations()
        check_tree(nb, oracle, s, pm, leaf, order, 0.5)


@pytest.mark.parametrize("n,leaf", [(1025, 1), (4097, 64), (16384, 17), (20001, 5)])
def test_dual_records_at_block_edges(nb, oracle, n, leaf):
    pm, _ = nb.scenarios.hernquist(n, seed=n)
    with dual_solver(nb, pm, leaf, 0.5) as s:
        s.update_accelerations()
        check_dual_tree(nb, oracle, s, pm, leaf)
