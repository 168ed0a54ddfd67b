"""The FP64 block GEMM on a right operand whose columns are strided (its last leg is contracted), at the edges of its
tiles and in every storage order of the contracted legs."""
import numpy as np
import pytest

from tests.test_gpu_gemm_f64 import check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N", [(1, 1), (9, 15), (16, 16), (17, 17), (31, 33), (32, 32), (100, 49), (49, 100), (8, 70),
                                 (70, 8), (810, 800)])
@pytest.mark.parametrize("K", [1, 5, 48])
def test_tile_edges(M, N, K):
    rng = np.random.default_rng(M * 1000 + N + K)
    x, y = rng.standard_normal((M, K)), rng.standard_normal((N, K))
    check(x, y, [1], [1])
    check(np.ascontiguousarray(x.T), y, [0], [1])


@pytest.mark.parametrize("order", [(0, 1, 2), (0, 2, 1), (1, 0, 2), (2, 0, 1)])
def test_contracted_legs_in_any_order(order):
    rng = np.random.default_rng(8)
    y = np.ascontiguousarray(rng.standard_normal((37, 6, 7)).transpose(order))
    check(rng.standard_normal((40, 6, 7)), y, [1, 2], [order.index(1), order.index(2)])
