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
