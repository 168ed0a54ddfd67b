"""The FLOPs that the statistics book for a decomposition's stages are those of what ran: sweeps, factorisation,
refinement."""
import numpy as np
import pytest

import quantit_gb300 as q
from tests.test_gpu_lq import graded, sectors

pytestmark = pytest.mark.gpu


def booked(mats, mode, cutoff=None):
    """(FP32, FP64 work), (FP32, FP64 sweeps) of one decomposition."""
    t = sectors(mats)
    q.set_gemm_mode(mode)
    q.stats.enable(True)
    try:
        q.stats.reset()
        q.linalg.svd(t, 1) if cutoff is None else q.linalg.svd(t, 1, cutoff, min_size=1, max_size=10 ** 6)
        work = [q.stats.get(k)["work"] for k in ("jacobi_fp32", "jacobi_fp64")]
    finally:
        q.stats.enable(False)
        q.set_gemm_mode("f64")
    return work, [q.linalg.last_svd_sweeps(fp32_stage=True), q.linalg.last_svd_sweeps()]


def sweeps(mats, n):
    return sum(s * (4.0 * max(a.shape) * min(a.shape) ** 2 + 3.0 * min(a.shape) ** 3) for s, a in zip(n, mats))


def factored(mats):
    return sum(min(a.shape) ** 2 * (10 / 3 * min(a.shape) + 4.0 * (max(a.shape) - min(a.shape))) for a in mats)


def test_plain_fp64():
    """Sectors of 48 columns and more are factored, tall ones (1.5 : 1 and more) if their rows are graded."""
    rng = np.random.default_rng(96)
    mats = [rng.standard_normal((30, 20)), rng.standard_normal((90, 60)), rng.standard_normal((60, 89)), graded(rng, 70, 120, 6)]
    work, n = booked(mats, "f64")
    assert work == [0.0, pytest.approx(sweeps(mats, n[1]) + factored(mats[2:]))]


def test_plain_split():
    rng = np.random.default_rng(97)
    mats = [rng.standard_normal((30, 20)), rng.standard_normal((70, 90))]
    work, n = booked(mats, "tf32x3")
    fp64 = sum(2.0 * min(a.shape) ** 3 + 2.0 * a.size * min(a.shape) for a in mats)
    assert work[0] == pytest.approx(sweeps(mats, n[0]) + sum(4.0 * min(a.shape) ** 3 for a in mats))
    assert work[1] == pytest.approx(sweeps(mats, n[1]) + fp64)


def test_resolved_anew():
    """A truncation below FP32's resolution: factored sweeps in FP64, no refinement."""
    rng = np.random.default_rng(98)
    mats = [graded(rng, 60, 60, 14)]
    work, n = booked(mats, "tf32x3", 1e-12)
    assert work[0] == pytest.approx(sweeps(mats, n[0]) + factored(mats))
    assert work[1] == pytest.approx(sweeps(mats, n[1]) + factored(mats))
