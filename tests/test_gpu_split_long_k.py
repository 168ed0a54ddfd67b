"""One output tile of the split-precision GEMM over a K that takes longer than a bounded wait on an mbarrier."""
import numpy as np
import pytest

import quantit_gb300 as q
from quantit_gb300.conserved import Z

pytestmark = pytest.mark.gpu


def test_long_contraction():
    """Alternating signs: every partial sum is a small integer, so FP32 accumulation is exact."""
    K = 2 ** 27 + 3
    y = np.ones((K, 1))
    y[1::2] = -1.0
    y[-100:] = 1.0
    a = q.btensor([[(1, Z(0))], [(K, Z(0))]], Z(0)).set_blocks([((0, 0), np.ones((1, K)))])
    b = q.btensor([[(K, Z(0))], [(1, Z(0))]], Z(0)).set_blocks([((0, 0), y)])
    q.set_gemm_mode("tf32x3")
    try:
        got = a.tensordot(b, ([1], [0])).blocks()[0][1][0, 0]
    finally:
        q.set_gemm_mode("f64")
    assert got == y.sum()
