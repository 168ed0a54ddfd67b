"""The SVD of the split modes on sectors of any magnitude: its FP32 stage hands an orthogonal rotation to the FP64 one
whether the elements' squares are normal FP32 numbers, subnormal ones or zero."""
import numpy as np
import pytest

import quantit_gb300 as q
from tests.test_gpu_lq import graded, sectors

pytestmark = pytest.mark.gpu


def factors(mats, mode, cutoff=None):
    """{row charge: (U, values, V)} of the block-diagonal tensor of ``mats``."""
    q.set_gemm_mode(mode)
    try:
        t = sectors(mats)
        U, d, V = q.linalg.svd(t, 1) if cutoff is None else q.linalg.svd(t, 1, cutoff, min_size=1, max_size=10 ** 6)
    finally:
        q.set_gemm_mode("f64")
    ub, vb = {k[1]: (k[0], v) for k, v in U.blocks()}, {k[1]: v for k, v in V.blocks()}
    return {ub[k[0]][0]: (ub[k[0]][1], s, vb[k[0]]) for k, s in d.blocks()}


def check_sector(a, u, s, v, whole):
    """Values and product to 1e-13 p of the sector's own largest value, both factors isometric in every column."""
    want = np.linalg.svd(a, compute_uv=False)
    bound = 1e-13 * max(a.shape) * want[0]
    np.testing.assert_allclose(s, want[:len(s)], atol=bound, rtol=0)
    rest = 0.0 if whole else want[len(s)]
    assert np.linalg.norm((u * s) @ v.T - a, 2) <= rest + bound
    for f in (u, v):
        assert np.max(np.abs(f.T @ f - np.eye(f.shape[1]))) < 1e-11


SCALES = [1.0, 1e-10, 1e-15, 1e-18, 1e-20, 1e-21, 1e-22, 1e-23, 1e-30, 1e-120, 1e15]


@pytest.mark.parametrize("mode", ["tf32x3", "bf16x3"])
@pytest.mark.parametrize("scale", SCALES)
def test_plain(scale, mode):
    rng = np.random.default_rng(61)
    mats = [scale * a for a in (rng.standard_normal((120, 62)), rng.standard_normal((50, 90)), graded(rng, 80, 64, 8),
                                graded(rng, 48, 48, 5), rng.standard_normal((9, 7)))]
    for i, (u, s, v) in factors(mats, mode).items():
        check_sector(mats[i], u, s, v, True)


@pytest.mark.parametrize("scale", SCALES[:-2])
def test_truncated_above_fp32_resolution(scale):
    rng = np.random.default_rng(62)
    mats = [scale * a / np.linalg.norm(a) for a in (graded(rng, 120, 80, 8), graded(rng, 70, 90, 9), graded(rng, 30, 20, 6))]
    out = factors(mats, "tf32x3", 1e-3 * scale)
    assert sorted(out) == [0, 1, 2]
    for i, (u, s, v) in out.items():
        assert 5 < len(s) < min(mats[i].shape)
        check_sector(mats[i], u, s, v, False)


def test_weak_sector_beside_a_normal_one():
    rng = np.random.default_rng(63)
    weak = 1e-21 * rng.standard_normal((70, 60))
    mats = [rng.standard_normal((80, 66)), weak, 1e-22 * graded(rng, 64, 64, 6)]
    for i, (u, s, v) in factors(mats, "tf32x3").items():
        check_sector(mats[i], u, s, v, True)
