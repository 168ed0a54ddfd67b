"""More sectors than one decomposition takes are refused with the same error whatever runs first."""
import numpy as np
import pytest

import quantit_gb300 as q
from quantit_gb300.conserved import Z, ZZ

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["f64", "tf32x3"])
def test_truncated(mode):
    n = 270
    charges = [ZZ(i, j) for i in range(n) for j in range(n)]
    inverse = [ZZ(-i, -j) for i in range(n) for j in range(n)]
    t = q.btensor([[(1, c) for c in charges], [(1, c) for c in inverse]], ZZ(0, 0))
    t.set_blocks([((i, i), np.ones((1, 1))) for i in range(n * n)])
    q.set_gemm_mode(mode)
    try:
        with pytest.raises(ValueError, match="too many sectors"):
            q.linalg.svd(t, 1, 1e-10)
    finally:
        q.set_gemm_mode("f64")


@pytest.mark.parametrize("mode", ["f64", "tf32x3"])
def test_batch(mode):
    t = q.btensor([[(70000, Z(0))], [(2, Z(0))], [(2, Z(0))]], Z(0))
    t.set_blocks([((0, 0, 0), np.random.default_rng(1).standard_normal((70000, 2, 2)))])
    q.set_gemm_mode(mode)
    try:
        with pytest.raises(ValueError, match="too many sectors"):
            q.linalg.svd(t)
        with pytest.raises(ValueError, match="too many sectors"):
            q.linalg.eigh(t)
    finally:
        q.set_gemm_mode("f64")
