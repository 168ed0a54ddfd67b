"""Contractions and decompositions whose planning tables are larger than a half of the staging ring (32 MB)."""
import numpy as np
import pytest

import quantit_gb300 as q
from quantit_gb300.conserved import Z

pytestmark = pytest.mark.gpu


def vector_blocks(n, x, first):
    """x as n blocks of one element: a row of blocks, or a column with ``first``."""
    leg, one = [(1, Z(0))] * n, [(1, Z(0))]
    t = q.btensor([leg, one] if first else [one, leg], Z(0))
    return t.set_blocks([((i, 0) if first else (0, i), x[i:i + 1].reshape(1, 1)) for i in range(n)])


def test_pairs_of_an_fp64_contraction():
    """840 x 840 output blocks: 45 MB of pairs, 23 MB of blocks, 11 MB of tiles; then as many pairs again."""
    rng = np.random.default_rng(81)
    n = 840
    a, b, v = rng.standard_normal(n), rng.standard_normal(n), rng.standard_normal(n)
    outer = vector_blocks(n, a, True).tensordot(vector_blocks(n, b, False), ([1], [0]))
    assert len(outer.block_indices()) == n * n
    got = outer.tensordot(vector_blocks(n, v, True), ([1], [0]))
    out = np.array([x[0, 0] for _, x in got.blocks()])
    want, room = a * np.dot(b, v), np.abs(a) * np.dot(np.abs(b), np.abs(v))
    assert np.all(np.abs(out - want) <= 2 * n * 2.0 ** -53 * room)


@pytest.mark.parametrize("mode", ["tf32x3", "bf16x3"])
def test_blocks_of_a_split_contraction(mode):
    """2 x 120000 operand blocks: 50 MB of block descriptors."""
    rng = np.random.default_rng(82)
    n = 120000
    a, b = rng.standard_normal(n), rng.standard_normal(n)
    q.set_gemm_mode(mode)
    try:
        got = vector_blocks(n, a, False).tensordot(vector_blocks(n, b, True), ([1], [0])).blocks()[0][1][0, 0]
    finally:
        q.set_gemm_mode("f64")
    # splits of 22 bits or more; FP32 accumulation of n terms
    assert abs(got - np.dot(a, b)) <= (2.0 ** -19 + 6 * n * 2.0 ** -23) * np.dot(np.abs(a), np.abs(b))


def test_tiles_of_an_fp64_contraction():
    """A 47000 x 47000 result: 33 MB of tiles."""
    rng = np.random.default_rng(83)
    n = 47000
    x, y, v = rng.standard_normal(n), rng.standard_normal(n), rng.standard_normal((n, 1))

    def one(z):
        return q.btensor([[(s, Z(0))] for s in z.shape], Z(0)).set_blocks([((0, 0), z)])
    outer = one(x.reshape(n, 1)).tensordot(one(y.reshape(1, n)), ([1], [0]))
    got = outer.tensordot(one(v), ([1], [0])).blocks()[0][1][:, 0]
    want, room = x * (y @ v[:, 0]), np.abs(x) * (np.abs(y) @ np.abs(v[:, 0]))
    assert np.all(np.abs(got - want) <= 2 * n * 2.0 ** -53 * room)
