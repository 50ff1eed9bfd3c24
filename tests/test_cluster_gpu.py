"""The two routes of the per-phase schedule: a small lattice's passes in one cluster, or
a launch per phase (set_cluster(False), and every larger lattice).  Each is held to the
reference's runs, to the oracle and to the wavefront; every test says which route it ran,
so that a moved limit cannot take a route its tests away."""
import numpy as np
import pytest

import pyoracle as po
import qcd_2d_gpu_b200 as q
from cases import CASES, SWEEPS
from conftest import load_case
from test_parity_gpu import FIELD_TOL, METRO_BITS_TOL, OBS_TOL, ORACLE_CASES, make

pytestmark = pytest.mark.gpu


def test_the_switch_and_what_it_reports():
    with q.Lattice(16, 16, 16, 6.0) as L:
        assert L.cluster()
        L.set_cluster(False)
        assert not L.cluster()
        L.set_cluster(True)
        assert L.cluster()
        L.set_schedule("wavefront")
        assert not L.cluster()
        L.set_schedule("phases")
        assert L.cluster()
    with q.Lattice(30, 34, 66, 6.0) as L:
        assert not L.cluster()
    assert q.load_library().qcd_set_cluster(None, 1) == -1
    assert q.load_library().qcd_get_cluster(None) == -1


@pytest.mark.parametrize("cluster", [True, False])
@pytest.mark.parametrize("name", list(CASES))
def test_fp64_reproduces_the_reference_on_both_routes(name, cluster):
    g = load_case(name)
    algo = g["case"][3]
    with make(g["case"]) as L:
        L.set_cluster(cluster)
        assert L.cluster() == cluster
        step = L.overrelax if algo == "or" else L.sweep
        obs = []
        for s in range(SWEEPS):
            step(1)
            obs.append(L.measure())
            if s == 0:
                f1 = L.store_config()
        fN, accept = L.store_config(), L.accept_counts()
    if algo == "metro":
        assert np.abs(f1 - g["field_1"]).max() <= METRO_BITS_TOL
        assert np.abs(fN - g["field_N"]).max() <= METRO_BITS_TOL
    else:
        assert np.array_equal(f1, g["field_1"]) and np.array_equal(fN, g["field_N"])
    assert np.abs(np.array(obs) - g["obs"]).max() <= OBS_TOL
    assert np.array_equal(accept, g["accept"])


@pytest.mark.parametrize("case", ORACLE_CASES, ids=lambda c: "_".join(map(str, c[:6])))
def test_fp64_phases_match_the_oracle(case):
    lt, lx, ly, algo, bc, hot, beta, eps, upd = case
    kw = dict(boundary=bc, epsilon=eps, upd=upd, seed=20261203)
    tape = q.rng_tape(kw["seed"], 0, lt * lx * ly // 2, 24 + SWEEPS * 6 * (4 * upd if algo == "metro" else 12) + 24)
    o = po.Oracle(lt, lx, ly, beta, algo=0 if algo == "metro" else 1, tape=tape, **kw)
    with q.Lattice(lt, lx, ly, beta, algo=algo, **kw) as L:
        L.set_cluster(False)
        assert not L.cluster()
        for x in (o, L):
            x.init_hot() if hot else x.init_cold()
            x.sweep(SWEEPS)
            x.overrelax(1)
        assert np.abs(L.store_config() - o.field()).max() <= FIELD_TOL
        assert np.array_equal(L.accept_counts(), o.accept())
    o.close()


# above the limit, rows of odd half length, last tiles partly empty
@pytest.mark.parametrize("dims", [(30, 34, 66), (6, 54, 62)], ids=lambda d: "x".join(map(str, d)))
@pytest.mark.parametrize("bc", [0, 1, 2])
@pytest.mark.parametrize("prec", ["fp64", "fp32"])
@pytest.mark.parametrize("algo", ["hb", "metro"])
def test_phases_equal_the_wavefront_at_every_boundary(dims, bc, prec, algo):
    out = []
    for mode in ("phases", "wavefront"):
        with q.Lattice(*dims, 7.0, algo=algo, boundary=bc, precision=prec, n_or=1, epsilon=0.3, upd=2,
                       renorm_every=1 if prec == "fp32" else 0, seed=31) as L:
            L.set_pair_layout(False)
            L.set_schedule(mode)
            assert not L.cluster()
            L.init_hot()
            L.sweep(3)
            L.overrelax(1)
            out.append((L.store_config(), L.accept_counts(), L.store_rng(), L.measure()))
    for x, y in zip(*out):
        assert np.array_equal(x, y)


# V/2 = 4, 240, 500, 1980, 3960, 4080
@pytest.mark.parametrize("dims", [(2, 2, 2), (8, 6, 10), (10, 10, 10), (18, 20, 22), (6, 34, 40)],
                         ids=lambda d: "x".join(map(str, d)))
@pytest.mark.parametrize("bc", [0, 1, 2])
@pytest.mark.parametrize("prec,algo", [("fp64", "hb"), ("fp64", "metro"), ("fp32", "hb"), ("fp32", "metro")])
def test_cluster_equals_the_phases(dims, bc, prec, algo):
    vh = dims[0] * dims[1] * dims[2] // 2
    out = []
    for cluster in (True, False):
        with q.Lattice(*dims, 7.0, algo=algo, boundary=bc, precision=prec, n_or=2, epsilon=0.3, upd=2,
                       renorm_every=2 if prec == "fp32" else 0, seed=5) as L:
            L.set_pair_layout(False)
            L.set_cluster(cluster)
            # (FP64 Metropolis leaves the cluster at 2048 sites)
            assert L.cluster() == (cluster and vh <= (2048 if (prec, algo) == ("fp64", "metro") else 4096))
            L.init_hot()
            L.sweep(3)
            L.overrelax(1)
            L.sweep(2)
            out.append((L.store_config(), L.accept_counts(), L.store_rng(), L.measure()))
    for x, y in zip(*out):
        assert np.array_equal(x, y)
