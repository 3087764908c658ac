"""The FP64 row kernel of the fused stage (32-wide tiles: per-cell
reconstruction, shuffles along i, edge warps, planned halo loads, the shock
points of the adaptive flux in a pass of their own) where it can go wrong:
extents at the edges of its tiles and k-chunks, every flux, first order,
limiter and clipping off, the uploaded sound speed in use, joined blocks.
Bit for bit against the CPU oracle."""
import numpy as np
import pytest

from eilmer4_b200 import workloads as W
from tests.parity import FLUX, assert_same

pytestmark = pytest.mark.gpu


def both(oracle, blocks, conns, flux, nsteps, tile, **kw):
    from eilmer4_b200.simcore import Simulation
    cfg = oracle.default_config(dimensions=3, flux_calculator=FLUX[flux], n_threads=0, **kw)
    ref = oracle.OracleSim(cfg)
    conf = {"dimensions": 3, "flux_calculator": flux}
    conf.update({k: (bool(v) if k != "interpolation_order" else v) for k, v in kw.items()})
    with Simulation(conf) as sim:
        for b in blocks:
            h = ref.add_block(b.ni, b.nj, b.nk, b.vtx, b.bc, b.inflow)
            ref.set_flow(h, b.prim)
            sim.upload(sim.add_block(b.ni, b.nj, b.nk, b.vtx, b.bc, b.inflow), b.prim)
        for c in conns:
            ref.connect(*c)
            sim.connect(*c)
        sim.set_tile(*tile)
        assert ref.run(nsteps) == 0
        sim.run(nsteps)
        for h in range(len(blocks)):
            gp, gc = sim.download(h)
            op, oc = ref.get_flow(h)
            assert_same(gc, oc, f"block {h} conserved, {flux}, tile {tile}")
            assert_same(gp[:8], op[:8], f"block {h} primitive, {flux}, tile {tile}")


def blast(ni, nj, nk, seed=5):
    """A block with flow through every face and a pressure jump inside it (shock
    points), its sound speeds uploaded an ulp off those of u."""
    b = W.inflow_3d_block(ni, nj, nk, seed, spacing=1.0 / 64.0)
    p = b.prim.reshape(8, nk, nj, ni)
    p[2] += 40.0 * np.sin(np.arange(nj))[None, :, None]
    p[3] -= 30.0 * np.cos(np.arange(nk))[:, None, None]
    hot = (slice(nk // 3, nk // 3 + 2), slice(nj // 3, nj // 3 + 2), slice(ni // 3, ni // 3 + 3))
    p[(6,) + hot] *= 6.0
    # T and p as update_thermo_from_rhou gives them (a first-order face takes
    # the cell's p, which this path forms from rho and u)
    Rgas = 8.31451 / 0.02896
    p[5] = p[6] * (1.0 / (Rgas / (1.4 - 1.0)))
    p[4] = p[0] * Rgas * p[5]
    p[7] = np.nextafter(np.sqrt(1.4 * Rgas * p[5]), 1.0e9)
    return b


@pytest.mark.parametrize("tile", [(32, 14, 32), (32, 8, 5), (32, 4, 8)])
@pytest.mark.parametrize("size", [(32, 14, 33), (33, 15, 2), (31, 13, 7), (65, 3, 9), (2, 2, 2)])
def test_extents_at_tile_edges(oracle, e4lib, size, tile):
    both(oracle, [blast(*size)], [], "hllc", 7, tile)


@pytest.mark.parametrize("flux", ["ausmdv", "hllc", "hanel", "adaptive_hanel_ausmdv"])
@pytest.mark.parametrize("tile", [(32, 14, 9), (32, 8, 32), (32, 4, 3)])
def test_fluxes(oracle, e4lib, flux, tile):
    both(oracle, [blast(37, 19, 11)], [], flux, 12, tile)


@pytest.mark.parametrize("kw", [{"interpolation_order": 1}, {"apply_limiter": 0},
                                {"extrema_clipping": 0}])
def test_options(oracle, e4lib, kw):
    b = blast(34, 17, 6)
    # (walls all round: a first-order face next to an inflow would take the
    # inflow state's own p, which this path forms from its rho and u)
    b.bc = (W.BC_SLIP_WALL,) * 6
    both(oracle, [b], [], "ausmdv", 6, (32, 14, 4), **kw)


@pytest.mark.parametrize("parts", [(2, 1, 1), (1, 3, 1), (2, 2, 2)])
@pytest.mark.parametrize("flux", ["hllc", "adaptive_hanel_ausmdv"])
def test_joined_blocks(oracle, e4lib, parts, flux):
    blocks, conns = W.split_block(blast(40, 30, 12), 3, parts)
    both(oracle, blocks, conns, flux, 10, (32, 14, 8))


def test_partial_tiles_cost_no_more_than_full_ones(e4lib):
    """125 cells in i fill the same four tiles as 128: the three idle lanes of
    the last tile must not slow its warps down (left with an unphysical state
    they took every face's plain divisions: 2.6 times the step)."""
    import torch

    from eilmer4_b200.simcore import Simulation

    def ms_per_step(ni):
        b = W.inflow_3d_block(ni, 112, 64, 5, spacing=1.0 / 64.0)
        with Simulation({"dimensions": 3, "flux_calculator": "ausmdv"}) as sim:
            sim.upload(sim.add_block(b.ni, b.nj, b.nk, b.vtx, b.bc, b.inflow), b.prim)
            sim.set_tile(32, 14, 16)
            sim.run(5)
            s = torch.cuda.ExternalStream(sim.stream_handle())
            best = 1.0e9
            for _ in range(3):
                e = [torch.cuda.Event(enable_timing=True) for _ in range(2)]
                e[0].record(s)
                sim.run(20)
                e[1].record(s)
                torch.cuda.synchronize()
                best = min(best, e[0].elapsed_time(e[1]) / 20)
            return best

    full, partial = ms_per_step(128), ms_per_step(125)
    assert partial < 1.4 * full, (partial, full)
