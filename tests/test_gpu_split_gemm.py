"""The split-precision tensor-core contraction at the edges of its split chunks, stages and tiles,
and over the leg orders its split kernel reads."""
import itertools

import numpy as np
import pytest

import quantit_gb300 as q
from quantit_gb300.conserved import Z

pytestmark = pytest.mark.gpu


@pytest.fixture(params=["tf32x3", "bf16x3"])
def mode(request):
    q.set_gemm_mode(request.param)
    yield request.param
    q.set_gemm_mode("f64")


def one_block(x):
    t = q.btensor([[(n, Z(0))] for n in x.shape], Z(0))
    return t.set_blocks([((0,) * x.ndim, x)])


def check(got, want, room, K):
    """Products of 22-bit (or longer) splits, up to 6 K of them accumulated in FP32."""
    assert np.all(np.abs(got - want) <= (2.0 ** -19 + 6 * K * 2.0 ** -23) * room)


def product(x, y, dx, dy):
    K = int(np.prod([x.shape[d] for d in dx]))
    got = one_block(x).tensordot(one_block(y), (dx, dy)).blocks()[0][1]
    check(got, np.tensordot(x, y, (dx, dy)), np.tensordot(np.abs(x), np.abs(y), (dx, dy)), K)


@pytest.mark.parametrize("M,N", [(1, 1), (7, 16), (8, 17), (129, 63), (64, 65), (127, 128), (260, 9), (3, 300)])
@pytest.mark.parametrize("K", [1, 8, 9, 16, 17, 31, 33, 64, 95])
def test_tile_and_chunk_edges(mode, M, N, K):
    rng = np.random.default_rng(M * 1000 + N + K)
    product(rng.standard_normal((M, K)), rng.standard_normal((K, N)), [1], [0])


def test_more_tiles_than_ctas(mode):
    rng = np.random.default_rng(2)
    product(rng.standard_normal((3000, 40)), rng.standard_normal((40, 2000)), [1], [0])


@pytest.mark.parametrize("dims", [(5, 1, 6, 3), (2, 7, 3, 4)])
def test_leg_orders(mode, dims):
    rng = np.random.default_rng(7)
    r1, r2, k1, k2 = dims
    x0, y0 = rng.standard_normal((r1, r2, k1, k2)), rng.standard_normal((k1, 3, k2, 2))
    for pa in itertools.permutations(range(4)):
        for pb in ((0, 2, 1, 3), (3, 0, 1, 2)):
            x, y = np.ascontiguousarray(x0.transpose(pa)), np.ascontiguousarray(y0.transpose(pb))
            product(x, y, [pa.index(2), pa.index(3)], [pb.index(0), pb.index(2)])
    x, y = rng.standard_normal((3, 2, 4, 5, 2, 3)), rng.standard_normal((4, 2, 3, 6, 2))
    product(x, y, [0, 2, 4], [2, 0, 4])


@pytest.mark.parametrize("sizes", [[1] * 40, [3, 9, 1, 17, 40, 2, 8, 16, 33], [64, 1, 1, 64, 1], [0, 5, 0, 0, 70, 0]])
def test_pairs_share_stages(mode, sizes):
    """An output block accumulated over many short pairs: several of them ride in one stage."""
    rng = np.random.default_rng(5)
    leg = [(s, Z(i)) for i, s in enumerate(sizes)]
    inv = [(s, c.inv()) for s, c in leg]
    n = len(sizes)
    a = q.btensor([[(150, Z(0)), (4, Z(n))], inv, leg], Z(0))
    b = q.btensor([leg, inv, [(20, Z(0))]], Z(0))
    ab = [((0, i, i), rng.standard_normal((150, s, s))) for i, s in enumerate(sizes)]
    bb = [((i, i, 0), rng.standard_normal((s, s, 20))) for i, s in enumerate(sizes)]
    got = a.set_blocks(ab).tensordot(b.set_blocks(bb), ([1, 2], [0, 1])).blocks()[0][1]
    want = sum(np.tensordot(x, y, ([1, 2], [0, 1])) for (_, x), (_, y) in zip(ab, bb))
    room = sum(np.tensordot(np.abs(x), np.abs(y), ([1, 2], [0, 1])) for (_, x), (_, y) in zip(ab, bb))
    check(got, want, room, sum(s * s for s in sizes))


def test_infinities_and_nan_pass_through(mode):
    """An operand with a non-finite value is not scaled; what it touches is non-finite, the rest is not."""
    rng = np.random.default_rng(9)
    x, y = rng.standard_normal((40, 24)), rng.standard_normal((24, 30))
    x[3, 5], x[17, 2] = np.inf, np.nan
    got = one_block(x).tensordot(one_block(y), ([1], [0])).blocks()[0][1]
    bad = np.zeros(40, bool)
    bad[[3, 17]] = True
    assert not np.isfinite(got[bad]).any()
    room = np.abs(x[~bad]) @ np.abs(y)
    check(got[~bad], x[~bad] @ y, room, 24)
