"""FP32 heat-bath where most first tries are rejected, and re-projection of links
at every distance from the group."""
import numpy as np
import pytest

import qcd_2d_gpu_b200 as q

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(4, 2, 2), (8, 6, 10), (16, 16, 16)])
@pytest.mark.parametrize("beta", [0.05, 0.3, 1.5])
def test_rejections_of_either_lane_match_the_unpaired_loop(dims, beta):
    # small beta: several tries per link, in lane 0, lane 1 or both.  Same draws
    # in both layouts, so links agree to float rounding (2e-5 per pass, as the
    # FP32 oracle checks) but for decisions that rounding moves, and what those
    # links feed later in the pass.
    fields = []
    for paired in (True, False):
        with q.Lattice(*dims, beta, boundary=2, precision="fp32", seed=19) as L:
            L.set_pair_layout(paired)
            L.init_hot()
            L.sweep(1)
            fields.append(L.store_config().reshape(-1, 4))
    d = np.abs(fields[0] - fields[1]).max(axis=1)
    assert np.abs((fields[0] ** 2).sum(axis=1) - 1).max() < 1e-5
    assert (d > 2e-5).sum() <= 64, (d > 2e-5).sum()


@pytest.mark.parametrize("lt", [4, 6])  # site pairs and planes
def test_reprojection_at_every_distance(lt):
    rng = np.random.default_rng(8)
    n = lt * 4 * 8 * 3
    u = rng.normal(size=(n, 4))
    u /= np.linalg.norm(u, axis=1, keepdims=True)
    off = np.array([0, 1e-7, -3e-7, 2e-6, 4.9e-6, 5.1e-6, -4.9e-6, -5.1e-6, 1e-4, -1e-3, 0.3, -0.7, 1e3, -1 + 1e-10])
    u = (u * (1 + off[np.arange(n) % len(off)])[:, None]).astype(np.float32).astype(np.float64)
    with q.Lattice(lt, 4, 8, 6.0, precision="fp32") as L:
        L.load_config(u)
        L.normalize()
        got = L.store_config().reshape(-1, 4)
    want = u / np.linalg.norm(u, axis=1, keepdims=True)
    # one rounding to single precision of values up to 1: half of 2^-24, and the
    # double-precision error of the scale on top, far below the other half
    assert np.abs(got - want).max() <= 2.0 ** -24
