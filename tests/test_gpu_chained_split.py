"""The chained split contractions of a bond update (the Hamiltonian times a two-site state, both environment
updates), which take an operand's scale from the GEMM that wrote it, against the same contractions made one by
one: equal to the last bit, at any magnitude, with empty products too."""
import numpy as np
import pytest

import quantit_gb300 as q
from quantit_gb300 import algorithms, networks

pytestmark = pytest.mark.gpu


def same(x, y):
    bx, by = x.blocks(), y.blocks()
    assert [k for k, _ in bx] == [k for k, _ in by]
    for (_, u), (_, v) in zip(bx, by):
        np.testing.assert_array_equal(u, v)


@pytest.mark.parametrize("mode", ["tf32x3", "bf16x3"])
@pytest.mark.parametrize("persistent", [True, False])
@pytest.mark.parametrize("D,scale", [(2, 1.0), (17, 1e-80), (70, 1e90), (300, 1.0), (40, 0.0)])
def test_chains(D, scale, persistent, mode):
    mpo = networks.heisenberg(20)
    mps = networks.random_bMPS(D, mpo, q.conserved.Z(0), seed=D)
    left, right = algorithms.environments(mpo, mps, [9])[9]
    left = left * scale
    theta = mps[9].tensordot(mps[10], ([2], [0]))
    H = algorithms.compute_2sites_hamil(mpo[9], mpo[10])
    q.set_gemm_mode(mode)
    q.set_persistent_gemm(persistent)
    try:
        got = algorithms.hamil2site_times_state(theta, H, left, right)
        x = left.tensordot(theta, ([0], [0])).tensordot(H, ([0, 2, 3], [0, 4, 5]))
        same(got, x.tensordot(right, ([1, 4], [0, 1])))
        got = algorithms.compute_left_env(mpo[9], mps[9], left)
        x = left.tensordot(mps[9], ([0], [0])).tensordot(mpo[9], ([0, 2], [0, 3]))
        same(got, x.tensordot(mps[9].conj(), ([0, 2], [0, 1])))
        got = algorithms.compute_right_env(mpo[10], mps[10], right)
        x = right.tensordot(mps[10], ([0], [2])).tensordot(mpo[10], ([0, 3], [2, 3]))
        same(got, x.tensordot(mps[10].conj(), ([3, 0], [1, 2])))
    finally:
        q.set_persistent_gemm(True)
        q.set_gemm_mode("f64")
