"""The plain sector SVD (identity start, exactly computed angles) against LAPACK in each GEMM mode, around
the register slices of its FP64 kernels (columns of 128, 256 and 512 elements)."""
import numpy as np
import pytest

import quantit_gb300 as q
from quantit_gb300.conserved import Z

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["f64", "tf32x3", "bf16x3"])
@pytest.mark.parametrize("m,n", [(1, 1), (7, 5), (128, 17), (129, 40), (65, 64), (257, 33), (513, 24)])
def test_svd_plain(m, n, mode):
    a = np.random.default_rng(m + n).standard_normal((m, n))
    t = q.btensor([[(m, Z(0))], [(n, Z(0))]], Z(0)).set_blocks([((0, 0), a)])
    q.set_gemm_mode(mode)
    try:
        U, d, V = q.linalg.svd_plain(t, 1, 1e-13)
    finally:
        q.set_gemm_mode("f64")
    u, s, v = (x.blocks()[0][1] for x in (U, d, V))
    want = np.linalg.svd(a, compute_uv=False)
    # FP64 sweeps whatever the mode: rounding of at most max(m, n) eps per value, and couplings of that
    # size are accepted
    tol = 8 * max(m, n, 8) * np.finfo(float).eps
    np.testing.assert_allclose(s, want, rtol=0, atol=tol * want[0])
    np.testing.assert_allclose((u * s) @ v.T, a, rtol=0, atol=tol * want[0])
    for f in (u, v):
        assert np.max(np.abs(f.T @ f - np.eye(len(s)))) < tol
