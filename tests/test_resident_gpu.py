"""Small lattices, whose passes run in one cluster (links in shared memory), around
the sizes where that begins and ends: up to 4096 sites of a parity or site pairs
(Metropolis 2048, but 4096 on FP32 planes).  Exact comparisons."""
import numpy as np
import pytest

import qcd_2d_gpu_b200 as q

pytestmark = pytest.mark.gpu

# V/2 = 4, 15 * 16 (last slots empty), 512, 2048, 2052, 3960, 4096, 4104
DIMS = [(2, 2, 2), (6, 8, 10), (10, 10, 10), (16, 16, 16), (6, 18, 38), (18, 20, 22), (2, 64, 64), (6, 36, 38)]


@pytest.mark.parametrize("dims", DIMS, ids=lambda d: "x".join(map(str, d)))
@pytest.mark.parametrize("bc", [0, 1, 2])
@pytest.mark.parametrize("prec,algo", [("fp64", "hb"), ("fp64", "metro"), ("fp32", "hb"), ("fp32", "metro")])
def test_cluster_equals_the_wavefront(dims, bc, prec, algo):
    out = []
    for mode in ("phases", "wavefront"):
        with q.Lattice(*dims, 7.0, algo=algo, boundary=bc, precision=prec, n_or=1, epsilon=0.3, upd=2,
                       renorm_every=2 if prec == "fp32" else 0, seed=5) as L:
            L.set_pair_layout(False)
            L.set_schedule(mode)
            L.init_hot()
            L.sweep(3)
            L.overrelax(1)
            L.sweep(2)
            out.append((L.store_config(), L.accept_counts(), L.store_rng(), L.measure()))
    for x, y in zip(*out):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("dims", [(4, 2, 2), (8, 6, 10), (16, 16, 32), (16, 18, 30), (16, 32, 32), (16, 30, 36)], ids=lambda d: "x".join(map(str, d)))
@pytest.mark.parametrize("algo", ["hb", "metro"])
def test_pairs_do_not_depend_on_the_split_into_launches(dims, algo):
    # 84 passes in one call (more than a launch takes) and in 21 calls
    out = []
    for calls in (1, 21):
        with q.Lattice(*dims, 6.0, algo=algo, boundary=2, precision="fp32", n_or=3, renorm_every=1, epsilon=0.3, upd=2,
                       seed=9) as L:
            assert L.pair_layout()
            L.init_hot()
            for _ in range(calls):
                L.sweep(21 // calls)
            out.append((L.store_config(), L.accept_counts(), L.store_rng()))
    for x, y in zip(*out):
        assert np.array_equal(x, y)
