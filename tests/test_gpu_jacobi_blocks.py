"""The FP64 sector Jacobi at the edges of its column blocks (widths 4 and 8, cut into equal blocks up to 64
rows) and of its register slices (32, 64 and 96 rows): svd and eigh against LAPACK."""
import numpy as np
import pytest

import quantit_gb300 as q
from quantit_gb300.conserved import Z

pytestmark = pytest.mark.gpu

EPS = np.finfo(float).eps


def tensor(mats):
    t = q.btensor([[(a.shape[0], Z(i)) for i, a in enumerate(mats)],
                   [(a.shape[1], Z(-i)) for i, a in enumerate(mats)]], Z(0))
    return t.set_blocks([((i, i), a) for i, a in enumerate(mats)])


@pytest.mark.parametrize("rows", [20, 32, 33, 64, 65, 97])
@pytest.mark.parametrize("cols", [(1, 2, 3), (5, 6, 7, 8), (9, 11, 13, 15), (16, 17, 20), (24, 25, 31), (33, 41, 47)])
def test_svd_blocks(rows, cols):
    rng = np.random.default_rng(rows + sum(cols))
    mats = [rng.standard_normal((max(rows, n), n)) for n in cols]
    for _ in range(4):  # both block widths are tried before one is kept
        U, d, V = q.linalg.svd(tensor(mats), 1)
        for (_, u), (_, s), (_, v), a in zip(U.blocks(), d.blocks(), V.blocks(), mats):
            # couplings of up to rows eps are accepted, and every value carries rounding of that order
            tol = 8 * max(a.shape[0], 8) * EPS
            want = np.linalg.svd(a, compute_uv=False)
            np.testing.assert_allclose(s, want, rtol=0, atol=tol * want[0])
            np.testing.assert_allclose((u * s) @ v.T, a, rtol=0, atol=tol * want[0])
            for f in (u, v):
                assert np.max(np.abs(f.T @ f - np.eye(f.shape[1]))) < tol


@pytest.mark.parametrize("sizes", [(1, 2, 3, 5), (7, 8, 9, 11), (15, 16, 17), (31, 32, 33), (63, 64, 65), (96, 97)])
def test_eigh_blocks(sizes):
    rng = np.random.default_rng(sum(sizes))
    mats = [a + a.T for a in (rng.standard_normal((n, n)) for n in sizes)]
    for _ in range(4):
        d, U = q.linalg.eigh(tensor(mats))
        for (_, w), (_, u), a in zip(d.blocks(), U.blocks(), mats):
            # the columns are shifted by the Frobenius norm, at most sqrt(n) times the largest value
            n = a.shape[0]
            tol = 16 * max(n, 8) * EPS * np.linalg.norm(a)
            np.testing.assert_allclose(np.sort(w), np.linalg.eigvalsh(a), rtol=0, atol=tol)
            np.testing.assert_allclose((u * w) @ u.T, a, rtol=0, atol=tol)
            assert np.max(np.abs(u.T @ u - np.eye(n))) < 8 * max(n, 8) * EPS
