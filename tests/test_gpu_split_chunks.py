"""The split-precision GEMM cuts K into chunks of 128 bytes in launches of no more tiles than SMs and of 64 in larger
ones: the same bits either way, at the edges of both."""
import numpy as np
import pytest

import quantit_gb300 as q
from quantit_gb300.conserved import Z
from tests.test_gpu_split_gemm import check, one_block

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["tf32x3", "bf16x3"])
@pytest.mark.parametrize("K", [1, 8, 15, 16, 17, 24, 31, 32, 33, 48, 63, 64, 65, 96, 97, 129, 200])
def test_few_tiles_and_many(mode, K):
    rng = np.random.default_rng(K)
    # at most 2 n tiles of 128 x 128 in the large product, 2 in the small one, whatever the number of SMs
    n = 400
    x, y = rng.uniform(-1, 1, (128 * n, K)), rng.uniform(-1, 1, (K, 140))
    x[0, 0], y[0, 0] = 1.5, 1.5  # the same scales
    q.set_gemm_mode(mode)
    try:
        large = one_block(x).tensordot(one_block(y), ([1], [0])).blocks()[0][1]
        small = one_block(x[:100]).tensordot(one_block(y), ([1], [0])).blocks()[0][1]
    finally:
        q.set_gemm_mode("f64")
    assert np.array_equal(large[:100], small)
    check(small, x[:100] @ y, np.abs(x[:100]) @ np.abs(y), K)


@pytest.mark.parametrize("mode", ["tf32x3", "bf16x3"])
@pytest.mark.parametrize("Ks", [(1,) * 9, (8, 16, 24, 32, 3, 40, 1), (24, 24, 24), (33, 7, 64, 1, 95, 17), (200, 1, 1, 1, 1, 31)])
def test_pairs_share_a_stage(mode, Ks):
    """Contracted sections of every length behind one another in an output block."""
    rng = np.random.default_rng(7)
    a, b = [rng.uniform(-1, 1, (30, k)) for k in Ks], [rng.uniform(-1, 1, (k, 77)) for k in Ks]
    a[0][0, 0] = b[0][0, 0] = 1.5
    sections = [(k, Z(0)) for k in Ks]
    out = []
    for m in (30, 60000):
        A = q.btensor([[(m, Z(0))], sections], Z(0))
        A.set_blocks([((0, i), np.concatenate([x, np.zeros((m - 30, x.shape[1]))])) for i, x in enumerate(a)])
        B = q.btensor([sections, [(77, Z(0))]], Z(0)).set_blocks([((i, 0), x) for i, x in enumerate(b)])
        q.set_gemm_mode(mode)
        try:
            out.append(A.tensordot(B, ([1], [0])).blocks()[0][1][:30])
        finally:
            q.set_gemm_mode("f64")
    assert np.array_equal(out[0], out[1])
    check(out[0], sum(x @ y for x, y in zip(a, b)), sum(np.abs(x) @ np.abs(y) for x, y in zip(a, b)), sum(Ks))
