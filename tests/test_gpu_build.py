"""The tree build at the edges of its climb blocks (128 to 4096 Karras nodes by size and leaf) and of its prefix
scans (one kernel up to eight 2048-position tiles, two above): every node record bit-exact against the oracle."""
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


@pytest.mark.parametrize("n,leaf", [(257, 1), (1027, 1), (1700, 17), (2050, 16), (4097, 41), (4098, 41), (98_303, 1), (98_305, 5), (200_003, 2), (400_001, 4), (800_003, 16),
                                    (1_600_001, 32)])
def test_records_by_block_size(nb, oracle, n, leaf):
    pm, _ = nb.scenarios.plummer(n, seed=n)
    with make_solver(nb, pm, order=2, leaf=leaf) as s:
        s.update_accelerations_async()
        check_tree(nb, oracle, s, pm, leaf, 2, 0.5)


@pytest.mark.parametrize("n,leaf", [(49_153, 64), (100_003, 16), (200_001, 17), (400_001, 16), (800_003, 64)])
def test_dual_records_by_block_size(nb, oracle, n, leaf):
    pm, _ = nb.scenarios.hernquist(n, seed=n)
    with dual_solver(nb, pm, leaf, 0.5) as s:
        s.update_accelerations_async()
        check_dual_tree(nb, oracle, s, pm, leaf)
