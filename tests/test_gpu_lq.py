"""The LQ-preconditioned sector SVD against LAPACK at the edges of its panels (8 reflections), with
and without a truncation, and on the matrices a factorisation can go wrong on."""
import numpy as np
import pytest

import quantit_gb300 as q
from quantit_gb300.conserved import Z

pytestmark = pytest.mark.gpu


def sectors(mats):
    t = q.btensor([[(a.shape[0], Z(i)) for i, a in enumerate(mats)],
                   [(a.shape[1], Z(-i)) for i, a in enumerate(mats)]], Z(0))
    return t.set_blocks([((i, i), a) for i, a in enumerate(mats)])


def check(mats, truncated, mode):
    """Values to 1e-13 p of the largest, factors that multiply back and are isometric to 1e-12."""
    t = sectors(mats)
    q.set_gemm_mode(mode)
    try:
        U, d, V = q.linalg.svd(t, 1, 1e-300, min_size=1, max_size=10 ** 6) if truncated else q.linalg.svd(t, 1)
    finally:
        q.set_gemm_mode("f64")
    # the new leg has one section per sector, in charge order of the row leg
    dv = {k[0]: v for k, v in d.blocks()}
    ub, vb = {k[1]: (k[0], v) for k, v in U.blocks()}, {k[1]: v for k, v in V.blocks()}
    seen = set()
    for s, val in dv.items():
        i, u = ub[s]
        v = vb[s]
        a = mats[i]
        want = np.linalg.svd(a, compute_uv=False)
        top = max(want[0], 1e-300)
        assert np.all(np.diff(val) <= 0)
        np.testing.assert_allclose(val, want[:len(val)], atol=1e-13 * max(a.shape) * top, rtol=0)
        np.testing.assert_allclose((u * val) @ v.T, a, atol=1e-13 * max(a.shape) * top, rtol=0)
        good = val > 1e-12 * top
        for f in (u[:, good], v[:, good]):
            assert np.max(np.abs(f.T @ f - np.eye(f.shape[1]))) < 1e-11
        seen.add(i)
    assert seen == {i for i, a in enumerate(mats) if truncated is False or np.any(a)}


def graded(rng, m, n, decades):
    r = 10.0 ** (-decades / 2 * np.arange(m) / m)
    c = 10.0 ** (-decades / 2 * np.arange(n) / n)
    return rng.permutation(r)[:, None] * rng.standard_normal((m, n)) * rng.permutation(c)


@pytest.mark.parametrize("truncated,mode", [(True, "f64"), (False, "f64"), (True, "tf32x3")])
def test_panel_edges(truncated, mode):
    rng = np.random.default_rng(41)
    shapes = [(12, 12), (13, 12), (17, 16), (16, 17), (25, 24), (70, 33), (40, 41), (48, 48), (50, 49), (49, 55),
              (57, 56), (90, 57), (64, 65), (11, 30), (1, 5), (300, 130)]
    check([graded(rng, m, n, 10) for m, n in shapes], truncated, mode)


@pytest.mark.parametrize("mode", ["f64", "tf32x3"])
def test_difficult_sectors(mode):
    rng = np.random.default_rng(43)
    rank5 = rng.standard_normal((80, 5)) @ rng.standard_normal((5, 60))
    zero_rows = graded(rng, 70, 64, 6)
    zero_rows[::3] = 0.0
    equal = np.linalg.qr(rng.standard_normal((64, 64)))[0]           # all values equal
    diagonal = np.diag(10.0 ** -np.linspace(0, 13, 50))[rng.permutation(50)]
    tiny = 1e-120 * graded(rng, 60, 60, 8)
    check([rank5, zero_rows, equal, diagonal, rng.standard_normal((100, 100))], True, mode)
    check([tiny], True, mode)


def test_nan_does_not_spread_between_sectors():
    """A sector with a NaN neither hangs nor faults, and leaves the other sectors alone."""
    rng = np.random.default_rng(44)
    a, b = graded(rng, 60, 50, 6), graded(rng, 60, 50, 6)
    b[3, 4] = np.nan
    U, d, V = q.linalg.svd(sectors([a, b]), 1)
    vals = {k[0]: v for k, v in d.blocks()}
    want = np.linalg.svd(a, compute_uv=False)
    assert any(v.shape == want.shape and np.allclose(v, want, atol=1e-12 * want[0], rtol=0) for v in vals.values())
