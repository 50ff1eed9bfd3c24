"""Captured chains of phase launches: lattices above the cluster's limit, and small ones
with the cluster off, replay what the same calls do uncaptured.  The first launch of the
chain follows a kernel, a memset or the join of two streams, and a lattice's first sweep
may itself be captured."""
import numpy as np
import pytest

import qcd_2d_gpu_b200 as q

pytestmark = pytest.mark.gpu


def state(L):
    return (L.store_config(), *L.series_read(1), L.store_rng())


@pytest.mark.parametrize("before", ["kernel", "memset", "join"])
@pytest.mark.parametrize("first", [False, True], ids=["warm", "first-sweep"])
@pytest.mark.parametrize("dims,prec,cluster",
                         [((8, 6, 10), "fp64", False), ((8, 6, 10), "fp32", False), ((6, 10, 14), "fp32", False),
                          ((8, 6, 10), "fp64", True), ((8, 6, 10), "fp32", True),
                          ((30, 34, 66), "fp64", True), ((30, 34, 66), "fp32", True), ((32, 34, 66), "fp32", True)],
                         ids=lambda v: "x".join(map(str, v)) if isinstance(v, tuple) else None)
def test_captured_chain_replays_the_same_run(dims, prec, cluster, first, before):
    import torch

    def lattice():
        L = q.Lattice(*dims, 6.0, boundary=2, precision=prec, n_or=1, renorm_every=1 if prec == "fp32" else 0, seed=7)
        L.set_cluster(cluster)
        L.series_reserve(1)
        L.init_hot()
        if not first:
            L.sweep(1)
        return L

    with lattice() as a, lattice() as b:
        s, side = torch.cuda.Stream(), torch.cuda.Stream()
        x = torch.zeros(1024, device="cuda")
        b.set_stream(s.cuda_stream)
        torch.cuda.synchronize()
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            if before == "join":
                side.wait_stream(s)
                with torch.cuda.stream(side):
                    x += 1
                s.wait_stream(side)
            elif before == "memset":
                x.zero_()
            else:
                x += 1
            b.sweep(2)
            b.measure_into_series(0)
            b.overrelax(1)
        for _ in range(3):
            a.sweep(2)
            a.measure_into_series(0)
            a.overrelax(1)
            g.replay()
            torch.cuda.synchronize()
            for u, v in zip(state(a), state(b)):
                assert np.array_equal(u, v)
        # (asked last: a lattice whose first sweep is captured has not been asked before)
        assert a.cluster() == b.cluster() == (cluster and dims == (8, 6, 10))
        del g
        torch.cuda.synchronize()


# the sizes of the other chain tests, most of them below the cluster's limit
@pytest.mark.parametrize("dims", [(2, 2, 2), (6, 4, 2), (6, 10, 14), (10, 6, 26)], ids=lambda d: "x".join(map(str, d)))
@pytest.mark.parametrize("bc", [0, 1, 2])
@pytest.mark.parametrize("prec,algo", [("fp64", "hb"), ("fp64", "metro"), ("fp32", "hb"), ("fp32", "metro")])
def test_small_chained_phases_equal_one_persistent_launch(dims, bc, prec, algo):
    out = []
    for mode in ("phases", "wavefront"):
        with q.Lattice(*dims, 7.0, algo=algo, boundary=bc, precision=prec, n_or=2, epsilon=0.3, upd=2,
                       renorm_every=1 if prec == "fp32" else 0, seed=31) as L:
            L.set_pair_layout(False)
            L.set_schedule(mode)
            L.set_cluster(False)
            assert not L.cluster()
            L.init_hot()
            m = []
            for _ in range(4):
                L.sweep(5)
                m.append(L.measure())
            out.append((L.store_config(), L.accept_counts(), L.store_rng(), m))
    for x, y in zip(*out):
        assert np.array_equal(x, y)
