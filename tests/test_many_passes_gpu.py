"""Sweeps with more over-relaxation passes than one list of passes holds (64) are the
same as the passes one after another."""
import numpy as np
import pytest

import qcd_2d_gpu_b200 as q

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims,prec", [((4, 6, 8), "fp64"), ((6, 6, 8), "fp32"), ((32, 34, 66), "fp32")],
                         ids=["fp64", "fp32", "fp32-phases"])
@pytest.mark.parametrize("n_or", [62, 63, 64, 65, 128, 200])
def test_long_sweeps_equal_their_passes(dims, prec, n_or):
    out = []
    for split in (False, True):
        with q.Lattice(*dims, 6.0, boundary=2, precision=prec, n_or=0 if split else n_or, seed=4) as L:
            L.init_hot()
            for _ in range(2):
                L.sweep(1)
                if split:
                    L.overrelax(n_or)
            out.append((L.store_config(), L.store_rng()))
    for x, y in zip(*out):
        assert np.array_equal(x, y)


def test_long_sweeps_reproject_on_their_last_pass():
    with q.Lattice(6, 6, 8, 6.0, precision="fp32", n_or=100, renorm_every=1, seed=4) as L:
        L.init_hot()
        L.sweep(3)
        # re-projected as they were stored: rounding to single precision alone is left
        # (four components, each within 2^-25 of norm 1)
        assert abs(L.check_unitarity(2.0 ** -22) - 1.0) < 2.0 ** -22
