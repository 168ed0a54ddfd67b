"""The block-width autotuner keeps apart the FP64 kernels with exactly computed angles (svd_plain) and the others."""
import numpy as np
import pytest

import quantit_gb300 as q
from tests.test_gpu_lq import sectors

pytestmark = pytest.mark.gpu


def test_plain_sweeps_do_not_decide_for_the_others():
    rng = np.random.default_rng(95)
    t = sectors([rng.standard_normal((200, 5)) for _ in range(33)])
    line = "R=8 max_q<=2^3 nsec<=2^6"
    for _ in range(6):
        q.linalg.svd_plain(t, 1, 1e-12)
    report = q.autotune_report().splitlines()
    assert any(x.startswith("fp64 exact " + line) and "tuned;" in x for x in report)
    assert not any(x.startswith("fp64 " + line) for x in report)
    for _ in range(6):
        q.linalg.svd(t, 1)
    assert any(x.startswith("fp64 " + line) and "tuned;" in x for x in q.autotune_report().splitlines())
