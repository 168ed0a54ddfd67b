"""The FP64 block GEMM on either side of the line between its 16 x 16 and 32 x 32 tiles, in numbers of tiles and in the
contracted length, against the same product cut into pieces that lie well below it."""
import numpy as np
import pytest

from tests.test_gpu_gemm_f64 import one_block

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K", [(1000, 1001, 127), (1000, 1001, 128), (2144, 2144, 130), (2208, 2177, 130), (800, 777, 129)])
def test_pieces_of_the_product(M, N, K):
    """Sums run over K in order whatever the tile, so the bits are the same."""
    rng = np.random.default_rng(M + K)
    x, y = rng.standard_normal((M, K)), rng.standard_normal((K, N))
    whole = one_block(x).tensordot(one_block(y), ([1], [0])).blocks()[0][1]
    rows, cols = [0, 31, M // 2, M - 40, M], [0, 17, N // 3, N - 33, N]
    for r0, r1 in zip(rows, rows[1:]):
        for c0, c1 in zip(cols, cols[1:]):
            r1, c1 = min(r1, r0 + 300), min(c1, c0 + 300)
            part = one_block(np.ascontiguousarray(x[r0:r1])).tensordot(one_block(np.ascontiguousarray(y[:, c0:c1])), ([1], [0]))
            assert np.array_equal(part.blocks()[0][1], whole[r0:r1, c0:c1])
    np.testing.assert_allclose(whole, x @ y, atol=2 * K * 2.0 ** -53 * np.max(np.abs(x) @ np.abs(y)), rtol=0)
