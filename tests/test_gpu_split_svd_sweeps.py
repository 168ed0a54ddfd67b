"""The untruncated SVD of the split modes: its FP64 sweeps start from the refined FP32 rotation, whose columns are
orthogonal to about 1e-6, and end in two or three where a start from anything else takes eight."""
import numpy as np
import pytest

import quantit_gb300 as q
from tests.test_gpu_lq import check, graded, sectors

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["tf32x3", "bf16x3"])
@pytest.mark.parametrize("shape", [(47, 47), (48, 48), (96, 48), (50, 49), (200, 90), (62, 120), (150, 150)])
def test_few_fp64_sweeps(shape, mode):
    rng = np.random.default_rng(71)
    q.set_gemm_mode(mode)
    try:
        q.linalg.svd(sectors([rng.standard_normal(shape) for _ in range(3)]), 1)
        sweeps = list(q.linalg.last_svd_sweeps())
    finally:
        q.set_gemm_mode("f64")
    # couplings of 1e-6 take one sweep, those of close pairs of values a second, a third confirms
    assert len(sweeps) == 3 and max(sweeps) <= 3


@pytest.mark.parametrize("mode", ["tf32x3", "bf16x3"])
def test_factors(mode):
    rng = np.random.default_rng(72)
    shapes = [(1, 5), (17, 16), (47, 47), (48, 48), (50, 49), (49, 55), (90, 57), (64, 65), (130, 300)]
    check([graded(rng, m, n, 10) for m, n in shapes], False, mode)
    check([rng.standard_normal(s) for s in shapes], False, mode)


@pytest.mark.parametrize("width", [24, 60, 150])
def test_weak_sectors_discard_beside_a_strong_one(width):
    """The truncation's level lies above the FP32 resolution of graded sectors and below that of a stronger one
    without small values: the weak ones discard, the strong one needs two FP64 sweeps.  Seven and more if they are all
    decomposed anew."""
    rng = np.random.default_rng(73)
    weak = [graded(rng, width, width, 9) for _ in range(3)]
    weak = [a / np.linalg.norm(a) for a in weak]
    strong = np.linalg.qr(rng.standard_normal((width + 5, width)))[0] * np.linspace(300.0, 1000.0, width)
    q.set_gemm_mode("tf32x3")
    try:
        U, d, V = q.linalg.svd(sectors(weak + [strong]), 1, 1e-5, min_size=1, max_size=10 ** 6)
        sweeps = list(q.linalg.last_svd_sweeps())
    finally:
        q.set_gemm_mode("f64")
    assert max(sweeps) <= 5
    ub, vb = {k[1]: (k[0], x) for k, x in U.blocks()}, {k[1]: x for k, x in V.blocks()}
    kept = {ub[k[0]][0]: s for k, s in d.blocks()}
    for i, a in enumerate(weak + [strong]):
        want = np.linalg.svd(a, compute_uv=False)
        np.testing.assert_allclose(kept[i], want[:len(kept[i])], atol=1e-13 * len(a) * want[0], rtol=0)
        assert len(kept[i]) == width if i == 3 else 2 < len(kept[i]) < width
    for k, s in d.blocks():
        i, u = ub[k[0]]
        for f in (u, vb[k[0]]):
            assert np.max(np.abs(f.T @ f - np.eye(len(s)))) < 1e-11
