"""The MRG32k3a step at the ends of its ranges, against the recurrence in Python's
integers: state words exactly, links of the hot start (24 draws per stream) to
double rounding."""
import itertools

import numpy as np
import pytest

import qcd_2d_gpu_b200 as q

pytestmark = pytest.mark.gpu

M1, M2 = 4294967087, 4294944443


def step(s):
    x = (1403580 * s[1] - 810728 * s[0]) % M1
    y = (527612 * s[5] - 1370589 * s[3]) % M2
    z = (x - y) % M1 or M1
    return [s[1], s[2], x, s[4], s[5], y], z


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
def test_recurrence_at_extreme_states(prec):
    ends1 = [0, 1, 208, 2 ** 31, M1 - 209, M1 - 1]
    ends2 = [0, 1, 22852, 2 ** 31, M2 - 1]
    states = [list(s) for s in itertools.product(ends1, ends1, [0, M1 - 1], ends2, [7], ends2)]
    lt, lx, ly = 6, 10, 60
    vh = lt * lx * ly // 2
    assert len(states) == vh
    with q.Lattice(lt, lx, ly, 6.0, precision=prec) as L:
        words = L.store_rng()
        words[: 6 * vh] = np.array(states, dtype=np.uint32).T.reshape(-1)
        L.load_rng(words)
        L.init_hot()
        got = L.store_rng()[: 6 * vh].reshape(6, vh).T
        field = L.store_config().reshape(2, vh, 3, 4)
    want = np.empty((2, vh, 3, 4))
    for i, s in enumerate(states):
        for k in range(24):
            s, z = step(s)
            want[k // 12, i, k // 4 % 3, k % 4] = z / M1 - 0.5
        assert got[i].tolist() == s, i
    want /= np.linalg.norm(want, axis=-1, keepdims=True)
    # z (1/m1) against z/m1: 2^-53 of values up to 1; normalised by at least 0.01
    # here, and rounded to single precision in an FP32 lattice
    assert np.abs(field - want).max() < (1e-13 if prec == "fp64" else 2.0 ** -24)
