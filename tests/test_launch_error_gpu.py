"""A launch that CUDA refuses is reported by the call that made it, and by no later
one: the runtime's record of the last error does not outlive the call."""
import pytest

import qcd_2d_gpu_b200 as q

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
def test_a_refused_launch_is_reported_once(prec):
    import torch

    # more t-slice pairs than a grid has rows (65535): the launch is refused on the host
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


def test_a_graph_refused_inside_a_capture_is_reported_once():
    # a batch that runs as graphs of its own cannot be captured: its streams are already
    # being captured when it begins
    import torch

    def batch():
        b = q.Batch([dict(lt=4, lx=4, ly=6 + 2 * i, beta=5.0, hot=1) for i in range(4)], precision="fp32")
        b.reserve(8)
        b.init()
        return b

    b, s = batch(), torch.cuda.Stream()
    b.set_stream(s.cuda_stream)
    b.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=s):
        torch.zeros(8, device="cuda").add_(1)
        with pytest.raises(q.QcdError) as e:
            b.run(2, measure_every=1)
    assert e.value.status == -2
    other = batch()  # nothing of the failure is left
    other.set_groups(1)
    other.run(2, measure_every=1)
    assert other.measured() == 2
    with q.Lattice(4, 4, 4, 6.0) as L:
        L.init_cold()
        L.sweep(1)
        L.normalize()
    del g
    torch.cuda.synchronize()
