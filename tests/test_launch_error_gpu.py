"""A launch that CUDA refuses is reported by the call that made it, and by no later
one: the runtime's record of the last error does not outlive the call.  Lt = 262160
wants more t-slice pairs than a grid has rows (65535), which the launch itself
refuses on the host."""
import pytest

import qcd_2d_gpu_b200 as q

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
def test_a_refused_launch_is_reported_once(prec):
    import torch

    with q.Lattice(262160, 2, 2, 6.0, precision=prec) as L, q.Lattice(4, 4, 4, 6.0, precision=prec) as other:
        L.init_cold()
        for call in (L.sweep, L.overrelax):
            with pytest.raises(q.QcdError) as e:
                call(1)
            assert e.value.status == -2
            other.init_cold()  # nothing of the failure is left for other calls and handles
            other.normalize()
            L.normalize()
            torch.zeros(8, device="cuda").add_(1)
        assert L.measure()[1] == pytest.approx(1.0, abs=1e-12)
        L.check_unitarity(0.0)
