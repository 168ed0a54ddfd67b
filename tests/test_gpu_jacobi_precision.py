"""Rounding errors of the FP64 block Jacobi where no factorisation spares it sweeps: no larger than those of plain
rotations (x' = c x - s y, y' = s x + c y in half-angle form, every one of them), which are the figures below."""
import numpy as np
import pytest

import quantit_gb300 as q
from quantit_gb300.conserved import Z

pytestmark = pytest.mark.gpu


@pytest.fixture(autouse=True)
def one_block_width():
    q.set_autotune(False)
    yield
    q.set_autotune(True)


def one_sector(a):
    return q.btensor([[(n, Z(0))] for n in a.shape], Z(0)).set_blocks([((0, 0), a)])


@pytest.mark.parametrize("p,n,plain", [(150, 40, 1.10e-15), (300, 45, 1.17e-15), (600, 45, 1.18e-15)])
def test_product_of_the_factors(p, n, plain):
    """||U d V^T - A|| / ||A|| of Gaussian matrices, the mean over six (2 % apart from each other)."""
    errors = []
    for seed in range(6):
        a = np.random.default_rng(seed).standard_normal((p, n))
        U, d, V = (t.blocks()[0][1] for t in q.linalg.svd(one_sector(a), 1))
        errors.append(np.linalg.norm((U * d) @ V.T - a) / np.linalg.norm(a))
    assert np.mean(errors) <= 1.06 * plain


@pytest.mark.parametrize("n,plain", [(150, 2.73e-15), (300, 3.93e-15)])
def test_eigenvalues(n, plain):
    """Relative error of the eigenvalues of symmetric matrices, the mean over six (7 % apart from each other)."""
    errors = []
    for seed in range(6):
        x = np.random.default_rng(seed).standard_normal((n, n))
        a = (x + x.T) / np.sqrt(8 * n)
        want = np.linalg.eigvalsh(a)
        d, U = q.linalg.eigh(one_sector(a))
        errors.append(np.linalg.norm(d.blocks()[0][1] - want) / np.linalg.norm(want))
    assert np.mean(errors) <= 1.1 * plain


@pytest.mark.parametrize("exponent", [-480, -470, -460, -440, 0, 440, 470])
@pytest.mark.parametrize("p,n,decades", [(80, 60, 6), (60, 45, 0), (60, 30, 3)])
def test_any_magnitude(exponent, p, n, decades):
    """A power of two times a matrix has its factors, down to where squared norms come near the end of FP64's range."""
    rng = np.random.default_rng(3)
    a = rng.standard_normal((p, n)) * 10.0 ** (-decades * rng.permutation(n) / n)
    U, d, V = (t.blocks()[0][1] for t in q.linalg.svd(one_sector(a * 2.0 ** exponent), 1))
    d = d * 2.0 ** -exponent
    want = np.linalg.svd(a, compute_uv=False)
    np.testing.assert_allclose(d, want, atol=1e-13 * p * want[0], rtol=0)
    assert np.linalg.norm((U * d) @ V.T - a, 2) <= 1e-13 * p * want[0]
    for f in (U, V):
        assert np.max(np.abs(f.T @ f - np.eye(n))) < 1e-12
