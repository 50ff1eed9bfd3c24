"""Configurations through the device entry points: every double of the AoS layout
lands in the store and comes back unchanged (rounded once to single precision for
an FP32 lattice), for sizes around the 128 and 256 sites a CTA stages, from
buffers that are only 8-byte aligned.  Exact: no arithmetic is involved."""
import numpy as np
import pytest

import qcd_2d_gpu_b200 as q

pytestmark = pytest.mark.gpu

# V/2 = 4, 8 (V/4 = 4), 120, 420, 1584, 9240, 256 and 512 exactly, 16 * 2560
DIMS = [(2, 2, 2), (4, 2, 2), (4, 6, 10), (6, 10, 14), (8, 18, 22), (20, 14, 66), (4, 8, 16), (8, 8, 16), (20, 64, 64)]


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
@pytest.mark.parametrize("dims", DIMS, ids=lambda d: "x".join(map(str, d)))
def test_device_configuration_round_trip(dims, prec):
    import torch

    lib = q.load_library()
    with q.Lattice(*dims, 4.0, precision=prec) as L:
        g = torch.Generator("cuda").manual_seed(5)
        src = torch.randn(L.V * 12 + 1, generator=g, dtype=torch.float64, device="cuda")[1:]
        out = torch.zeros(L.V * 12 + 2, dtype=torch.float64, device="cuda")
        torch.cuda.synchronize()
        assert lib.qcd_load_config_device(L.handle, src.data_ptr()) == 0
        assert lib.qcd_store_config_device(L.handle, out[1:].data_ptr()) == 0
        torch.cuda.synchronize()
        want = src if prec == "fp64" else src.float().double()
        assert torch.equal(out[1:-1], want)
        assert out[0] == 0 and out[-1] == 0  # nothing written outside
        for layout in (True, False):  # site pairs and planes hold the same links
            L.set_pair_layout(layout)
            assert np.array_equal(L.store_config(), want.cpu().numpy())
