"""FP32 heat-bath on site pairs where nearly every try is rejected (small beta: up to
hundreds of tries per link, in lane 0, lane 1 or both), against the loop of one float4
plane per class.  From a cold start the first phase, the y links of the even sites, has
staple sums of exactly 4 in both layouts, and a pass leaves those links as that phase
made them: they hold its draws alone and are equal bit for bit."""
import numpy as np
import pytest

import qcd_2d_gpu_b200 as q

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cluster", [True, False])
@pytest.mark.parametrize("dims,beta", [(d, b) for d in [(4, 2, 2), (8, 6, 10), (16, 16, 16)]
                                       for b in [0.01, 0.05, 0.3, 1.5] if b > 0.01 or d == (4, 2, 2)])
def test_every_lane_redraws_as_the_unpaired_loop(dims, beta, cluster):
    fields = []
    for paired in (True, False):
        with q.Lattice(*dims, beta, boundary=2, precision="fp32", seed=19) as L:
            L.set_pair_layout(paired)
            L.set_cluster(cluster)
            assert L.pair_layout() == paired and L.cluster() == cluster
            L.init_cold()
            L.sweep(1)
            fields.append(L.store_config().reshape(2, -1, 3, 4))
    for f in fields:
        assert np.isfinite(f).all()
        assert np.abs((f ** 2).sum(axis=-1) - 1).max() < 1e-5
    first = [f[0, :, 0] for f in fields]  # even sites, y
    assert np.array_equal(*first)
    assert len(np.unique(first[0], axis=0)) == len(first[0])


# at beta 0.01 a try is accepted with probability 0.443 (2 beta |A|)^1.5: 0.01 at the cold
# start's |A| = 4, but 1e-4 for the staples below 0.2 that random links make, so the limit
# of 4096 tries is reached somewhere on a lattice of more than a few links
@pytest.mark.parametrize("paired", [True, False])
@pytest.mark.parametrize("dims", [(8, 6, 10), (16, 16, 16)], ids=lambda d: "x".join(map(str, d)))
def test_the_limit_of_tries_is_reported(dims, paired):
    with q.Lattice(*dims, 0.01, boundary=2, precision="fp32", seed=19) as L:
        L.set_pair_layout(paired)
        L.init_cold()
        L.sweep(1)
        with pytest.raises(q.QcdError) as e:
            L.measure()
        assert e.value.status == -4
