"""svd_plain computes its rotation angles exactly for columns of more than 512 elements too."""
import numpy as np
import pytest

import quantit_gb300 as q
from tests.test_gpu_lq import sectors

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("p", [512, 513, 768, 769, 1024, 1025, 1536, 1537])
def test_equal_values(p):
    rng = np.random.default_rng(p)
    want = np.repeat([3.0, 1.0, 0.5], 7)
    a = np.linalg.qr(rng.standard_normal((p, 21)))[0] * want @ np.linalg.qr(rng.standard_normal((21, 21)))[0]
    U, d, V = (x.blocks()[0][1] for x in q.linalg.svd_plain(sectors([a]), 1, 1e-12))
    np.testing.assert_allclose(d, want, atol=1e-13 * p * 3, rtol=0)
    np.testing.assert_allclose((U * d) @ V.T, a, atol=1e-13 * p * 3, rtol=0)
    for f in (U, V):
        assert np.max(np.abs(f.T @ f - np.eye(21))) < 1e-11


def test_kernel_of_long_columns():
    """The kernels with FP32 angles never run for it: the class by which their block width is tuned stays unknown."""
    rng = np.random.default_rng(99)
    t = sectors([rng.standard_normal((600, 5)) for _ in range(33)])
    for _ in range(2):
        q.linalg.svd_plain(t, 1, 1e-12)
    assert not any(x.startswith("fp64 R=20 max_q<=2^3 nsec<=2^6") for x in q.autotune_report().splitlines())
