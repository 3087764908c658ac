"""The fused stage's tile shape and k-chunk chosen for the blocks at hand
(until e4c_set_tile or e4c_autotune fixes them): whatever is chosen gives the
oracle's bits, a set shape stays, and a new context chooses again."""
import pytest

from eilmer4_b200 import workloads as W
from tests.parity import FLUX, assert_same

pytestmark = pytest.mark.gpu

SHAPES = {(32, 14), (32, 8), (32, 4), (16, 16), (16, 8)}


@pytest.mark.parametrize("sizes", [[(5, 4, 3)], [(40, 36, 30)], [(16, 100, 9)],
                                   [(96, 17, 50), (12, 60, 16), (33, 29, 12)]])
def test_chosen_tile(oracle, e4lib, sizes):
    from eilmer4_b200.simcore import Simulation
    blocks = [W.inflow_3d_block(*n, 3 + q, spacing=1.0 / 64.0) for q, n in enumerate(sizes)]
    ref = oracle.OracleSim(oracle.default_config(dimensions=3, flux_calculator=FLUX["ausmdv"],
                                                 n_threads=0))
    with Simulation({"dimensions": 3, "flux_calculator": "ausmdv"}) as sim:
        for b in blocks:
            ref.set_flow(ref.add_block(b.ni, b.nj, b.nk, b.vtx, b.bc, b.inflow), b.prim)
            sim.upload(sim.add_block(b.ni, b.nj, b.nk, b.vtx, b.bc, b.inflow), b.prim)
        ti, tj, kc = sim.get_tile()
        assert (ti, tj) in SHAPES and kc >= 1
        assert ref.run(8) == 0
        sim.run(8)
        assert sim.get_tile() == (ti, tj, kc)
        for h in range(len(blocks)):
            assert_same(sim.download(h)[1], ref.get_flow(h)[1], f"block {h}, tile {ti}x{tj}x{kc}")
        sim.set_tile(64, 4, 7)
        sim.run(1)
        assert sim.get_tile() == (64, 4, 7)
    with Simulation({"dimensions": 3, "flux_calculator": "ausmdv"}) as sim:
        for b in blocks:
            sim.upload(sim.add_block(b.ni, b.nj, b.nk, b.vtx, b.bc, b.inflow), b.prim)
        assert sim.get_tile() == (ti, tj, kc)


def test_choices_of_several_layouts(oracle, e4lib):
    """Layouts for which the model takes different shapes (a long narrow block,
    cubes, a flat one), each with the oracle's bits."""
    from eilmer4_b200.simcore import Simulation
    chosen = []
    for n in [(24, 24, 24), (7, 83, 120), (96, 96, 96), (120, 112, 40)]:
        b = W.inflow_3d_block(*n, 3, spacing=1.0 / 64.0)
        ref = oracle.OracleSim(oracle.default_config(dimensions=3, flux_calculator=FLUX["hllc"],
                                                     n_threads=0))
        ref.set_flow(ref.add_block(b.ni, b.nj, b.nk, b.vtx, b.bc, b.inflow), b.prim)
        with Simulation({"dimensions": 3, "flux_calculator": "hllc"}) as sim:
            sim.upload(sim.add_block(b.ni, b.nj, b.nk, b.vtx, b.bc, b.inflow), b.prim)
            chosen.append(sim.get_tile())
            assert ref.run(4) == 0
            sim.run(4)
            assert_same(sim.download(0)[1], ref.get_flow(0)[1], f"{n}, tile {chosen[-1]}")
    assert len({c[:2] for c in chosen}) >= 3, chosen


@pytest.mark.parametrize("sizes", [[(48, 96, 96), (48, 96, 96)], [(96, 96, 96)], [(112, 112, 114)],
                                   [(40, 88, 91)], [(16, 64, 48)] * 9])
def test_fp32_choice_keeps_the_edge_warp_kernel(e4lib, sizes):
    """16-wide tiles are another kernel with other rounding: whatever the layout,
    the FP32-flux form's own choice is 32 wide."""
    from eilmer4_b200.simcore import Simulation
    with Simulation({"dimensions": 3, "flux_calculator": "hllc"}, precision="fp32_flux") as sim:
        for n in sizes:
            b = W.inflow_3d_block(*n, 3, spacing=1.0 / 64.0)
            sim.upload(sim.add_block(b.ni, b.nj, b.nk, b.vtx, b.bc, b.inflow), b.prim)
        assert sim.get_tile()[0] == 32


def test_get_tile_does_not_wait(e4lib):
    """Asking for the automatic choice while the library's stream is busy."""
    import time

    import torch

    from eilmer4_b200.simcore import Simulation
    with Simulation({"dimensions": 3, "flux_calculator": "hllc"}) as sim:
        assert sim.get_tile() == (32, 8, 32)
        b = W.inflow_3d_block(40, 36, 30, 3, spacing=1.0 / 64.0)
        sim.upload(sim.add_block(b.ni, b.nj, b.nk, b.vtx, b.bc, b.inflow), b.prim)
        with torch.cuda.stream(torch.cuda.ExternalStream(sim.stream_handle())):
            torch.cuda._sleep(int(1.0e9))
        t0 = time.perf_counter()
        tile = sim.get_tile()
        waited = time.perf_counter() - t0
        sim.synchronize()
        slept = time.perf_counter() - t0
        sim.run(1)
        assert sim.get_tile() == tile
    assert waited < 0.5 * slept, (waited, slept)


def test_choice_costs_little_host_time(e4lib):
    """64 uneven blocks: the model's 60-odd pairs took 3.2 ms when every pair
    scheduled every work item, 0.6 with those no schedule can save skipped."""
    import time

    from eilmer4_b200.simcore import Simulation
    with Simulation({"dimensions": 3, "flux_calculator": "hllc"}) as sim:
        for b in W.batched_blocks(64).blocks:
            sim.add_block(b.ni, b.nj, b.nk, b.vtx, b.bc, b.inflow)
        times = []
        for _ in range(8):
            t0 = time.perf_counter()
            sim.get_tile()
            times.append(time.perf_counter() - t0)
    assert min(times) < 1.8e-3, times


@pytest.mark.parametrize("sizes", [[(24, 24, 24)], [(64, 64, 64)], [(48, 36, 40)] * 4])
@pytest.mark.parametrize("precision", ["fp64", "fp32_flux"])
def test_autotune_is_no_slower_than_the_choice(e4lib, sizes, precision):
    """The tuner times the pair it finds in use beside its own list (whose chunks
    start at 16 planes: alone it would end at three times the step on 24^3)."""
    import torch

    from eilmer4_b200.simcore import Simulation
    with Simulation({"dimensions": 3, "flux_calculator": "ausmdv"}, precision=precision) as sim:
        for n in sizes:
            b = W.inflow_3d_block(*n, 3, spacing=1.0 / 64.0)
            sim.upload(sim.add_block(b.ni, b.nj, b.nk, b.vtx, b.bc, b.inflow), b.prim)
        s = torch.cuda.ExternalStream(sim.stream_handle())

        def ms_per_step():
            sim.run(10)
            best = 1.0e9
            for _ in range(4):
                e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
                e[0].record(s)
                sim.run(50)
                e[1].record(s)
                torch.cuda.synchronize()
                best = min(best, e[0].elapsed_time(e[1]) / 50)
            return best

        untuned = ms_per_step()
        tile, _ = sim.autotune(5)
        assert sim.get_tile() == tile
        tuned = ms_per_step()
    assert tuned < 1.05 * untuned, (tile, tuned, untuned)
