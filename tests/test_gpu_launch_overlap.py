"""Overlapped launches must not spread the next stage's CTAs unevenly: the steps
run back to back take no longer than the stage kernels timed one by one."""
import pytest

from eilmer4_b200 import workloads as W

pytestmark = pytest.mark.gpu


def test_overlapped_stages_take_no_longer_than_single_ones(e4lib):
    """400 work items on SMs that hold more CTAs of this tile (with the next
    stage's CTAs placed during the one before: 1.11 times)."""
    import torch

    from eilmer4_b200.simcore import Simulation
    b = W.inflow_3d_block(160, 128, 160, 5, spacing=1.0 / 64.0)
    n = 20
    with Simulation({"dimensions": 3, "flux_calculator": "hllc"}, precision="fp32_flux") as sim:
        sim.upload(sim.add_block(b.ni, b.nj, b.nk, b.vtx, b.bc, b.inflow), b.prim)
        sim.set_tile(16, 16, 32)
        sim.run(5)
        single = min(sim.profile(n)["stage"][0] / n for _ in range(3))
        s = torch.cuda.ExternalStream(sim.stream_handle())
        step = 1.0e9
        for _ in range(3):
            e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
            e[0].record(s)
            sim.run(n)
            e[1].record(s)
            torch.cuda.synchronize()
            step = min(step, e[0].elapsed_time(e[1]) / n)
    assert step < 1.06 * single, (step, single)
