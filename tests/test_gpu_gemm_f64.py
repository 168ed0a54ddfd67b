"""The FP64 block GEMM at the edges of its tile classes and over the leg orders it reads in place."""
import itertools

import numpy as np
import pytest

import quantit_gb300 as q
from quantit_gb300.conserved import Z

pytestmark = pytest.mark.gpu


def one_block(x):
    t = q.btensor([[(n, Z(0))] for n in x.shape], Z(0))
    return t.set_blocks([((0,) * x.ndim, x)])


def check(x, y, dx, dy):
    """Against numpy, elementwise: a sum of K products is within K ulp of sum |x||y|."""
    want = np.tensordot(x, y, (dx, dy))
    room = np.tensordot(np.abs(x), np.abs(y), (dx, dy))
    K = int(np.prod([x.shape[d] for d in dx]))
    got = one_block(x).tensordot(one_block(y), (dx, dy)).blocks()[0][1]
    assert np.all(np.abs(got - want) <= 2 * max(K, 1) * 2.0 ** -53 * room)


@pytest.mark.parametrize("M,N", [(1, 1), (8, 63), (63, 8), (8, 64), (64, 8), (9, 64), (64, 9), (16, 16), (17, 16),
                                 (32, 33), (5, 257), (256, 3), (257, 8), (130, 70), (700, 650)])
@pytest.mark.parametrize("K", [1, 3, 4, 37])
def test_tile_edges(M, N, K):
    rng = np.random.default_rng(M * 1000 + N + K)
    check(rng.standard_normal((M, K)), rng.standard_normal((K, N)), [1], [0])


@pytest.mark.parametrize("dims", [(5, 1, 6, 3), (2, 7, 3, 4), (1, 1, 70, 9)])
def test_leg_orders(dims):
    """Every order of A(r1, r2, k1, k2) against two of B: from matrices that are read in place to
    legs that do not fold to two strides."""
    rng = np.random.default_rng(7)
    r1, r2, k1, k2 = dims
    x0 = rng.standard_normal((r1, r2, k1, k2))
    y0 = rng.standard_normal((k1, 3, k2, 2))
    for pa in itertools.permutations(range(4)):
        for pb in ((0, 2, 1, 3), (3, 0, 1, 2), (2, 1, 0, 3)):
            x, y = np.ascontiguousarray(x0.transpose(pa)), np.ascontiguousarray(y0.transpose(pb))
            check(x, y, [pa.index(2), pa.index(3)], [pb.index(0), pb.index(2)])


def test_three_contracted_strides_are_packed():
    rng = np.random.default_rng(3)
    x, y = rng.standard_normal((3, 2, 4, 5, 2, 3)), rng.standard_normal((4, 2, 3, 6, 2))
    check(x, y, [0, 2, 4], [2, 0, 4])


def test_pairs_accumulate_over_more_than_one_batch():
    """An output block with more pairs than are staged at a time."""
    rng = np.random.default_rng(5)
    n = 71
    leg = [(1 + i % 3, Z(i)) for i in range(n)]
    inv = [(s, c.inv()) for s, c in leg]
    a = q.btensor([[(9, Z(0))], leg, inv], Z(0))
    b = q.btensor([inv, leg, [(4, Z(0))]], Z(0))
    ab = [((0, i, i), rng.standard_normal((9, 1 + i % 3, 1 + i % 3))) for i in range(n)]
    bb = [((i, i, 0), rng.standard_normal((1 + i % 3, 1 + i % 3, 4))) for i in range(n)]
    got = a.set_blocks(ab).tensordot(b.set_blocks(bb), ([1, 2], [0, 1])).blocks()[0][1]
    want = sum(np.tensordot(x, y, ([1, 2], [0, 1])) for (_, x), (_, y) in zip(ab, bb))
    room = sum(np.tensordot(np.abs(x), np.abs(y), ([1, 2], [0, 1])) for (_, x), (_, y) in zip(ab, bb))
    assert np.all(np.abs(got - want) <= 2 * 4 * n * 2.0 ** -53 * room)
