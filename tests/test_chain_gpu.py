"""Chained phase launches: a launch is set up while its predecessor drains, so a
missed wait or a stale line would show as a wrong link.  Small and ragged
lattices, where several launches fit on the GPU side by side, over many
launches; exact comparisons."""
import numpy as np
import pytest

import qcd_2d_gpu_b200 as q

pytestmark = pytest.mark.gpu

# rows of odd length: neighbouring threads' links share 32-byte sectors across CTAs
DIMS = [(2, 2, 2), (6, 4, 2), (6, 10, 14), (10, 6, 26), (54, 62, 70), (30, 34, 66)]


@pytest.mark.parametrize("dims", DIMS, ids=lambda d: "x".join(map(str, d)))
@pytest.mark.parametrize("prec,algo", [("fp64", "hb"), ("fp64", "metro"), ("fp32", "hb"), ("fp32", "metro")])
def test_chained_phases_equal_one_persistent_launch(dims, prec, algo):
    # the wavefront runs the same updates in one persistent launch per chain of passes
    out = []
    for mode in ("phases", "wavefront"):
        with q.Lattice(*dims, 7.0, algo=algo, boundary=1, precision=prec, n_or=2, epsilon=0.3, upd=2,
                       renorm_every=1 if prec == "fp32" else 0, seed=31) as L:
            L.set_pair_layout(False)
            L.set_schedule(mode)
            L.init_hot()
            m = []
            for _ in range(4):
                L.sweep(5)
                m.append(L.measure())
            out.append((L.store_config(), L.accept_counts(), L.store_rng(), m))
    for x, y in zip(*out):
        assert np.array_equal(x, y)


@pytest.mark.parametrize("fork", [False, True])
@pytest.mark.parametrize("dims,prec", [((8, 6, 10), "fp32"), ((6, 10, 14), "fp32"), ((8, 6, 10), "fp64")])
def test_captured_chain_replays_the_same_run(dims, prec, fork):
    import torch

    def lattice():
        L = q.Lattice(*dims, 6.0, boundary=2, precision=prec, n_or=1, renorm_every=1 if prec == "fp32" else 0, seed=7)
        L.series_reserve(4)
        L.init_hot()
        L.sweep(1)
        return L

    a, b = lattice(), lattice()
    want = []
    for _ in range(3):
        a.sweep(2)
        a.measure_into_series(0)
        want.append((a.store_config(), a.series_read(1), a.store_rng()))
    s, side = torch.cuda.Stream(), torch.cuda.Stream()
    x = torch.zeros(1024, device="cuda")
    b.set_stream(s.cuda_stream)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        if fork:  # the first launch of the chain follows a join of two streams
            side.wait_stream(s)
            with torch.cuda.stream(side):
                x += 1
            x.mul_(1)
            s.wait_stream(side)
        b.sweep(2)
        b.measure_into_series(0)
    for w in want:
        g.replay()
        torch.cuda.synchronize()
        got = (b.store_config(), b.series_read(1), b.store_rng())
        for u, v in zip(got, w):
            assert np.array_equal(u, v)
    assert x[0].item() == (3 if fork else 0)
    del g
    torch.cuda.synchronize()
    a.close()
    b.close()
