"""The truncating SVD of the split modes with a sector too wide for the FP64 factorisation (about 1590 columns)."""
import numpy as np
import pytest

import quantit_gb300 as q
from tests.test_gpu_lq import sectors

pytestmark = pytest.mark.gpu


def test_wide_sector_keeps_its_fp32_rotation():
    """A wide sector beside one whose norm puts the truncation below its FP32 resolution: the wide one discards its
    columns below the threshold and takes a sweep to decouple the others and a few among them; from the identity
    its kept columns alone would take ten and more."""
    rng = np.random.default_rng(91)
    n = 1600
    values = 10.0 ** (-8.0 * (np.arange(n) / n) ** 0.3)
    u, v = (np.linalg.qr(rng.standard_normal((n, n)))[0] for _ in range(2))
    wide = (u * values) @ v.T
    strong = 1e3 * rng.standard_normal((30, 24))
    cutoff = 4e-6 * np.sqrt(n)
    q.set_gemm_mode("tf32x3")
    try:
        U, d, V = q.linalg.svd(sectors([wide, strong]), 1, cutoff, min_size=1, max_size=10 ** 6)
        sweeps = list(q.linalg.last_svd_sweeps())
    finally:
        q.set_gemm_mode("f64")
    s = dict((k[0], x) for k, x in d.blocks())
    rows = {k[1]: k[0] for k, _ in U.blocks()}
    got = {rows[k]: x for k, x in s.items()}
    assert 100 < len(got[0]) < n - 100 and len(got[1]) == 24
    np.testing.assert_allclose(got[0], values[:len(got[0])], atol=1e-13 * n, rtol=0)
    np.testing.assert_allclose(got[1], np.linalg.svd(strong, compute_uv=False), atol=1e-13 * 30 * 1e4, rtol=0)
    assert max(sweeps) <= 6
