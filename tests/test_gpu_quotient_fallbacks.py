"""States that the batched quotients leave to plain divisions: divisors with the
top 20 mantissa bits set, ordinary values of a density, a pressure, a sound
speed, a velocity or a limiter's sum of squares.  A block whose every cell is one,
bit for bit against the CPU oracle on each kernel that forms quotients."""
import math

import numpy as np
import pytest

from eilmer4_b200 import workloads as W
from tests.test_gpu_fused_rows import both

pytestmark = pytest.mark.gpu

RGAS = 8.31451 / 0.02896
CV = RGAS / 0.4
ALMOST = 1.0 - 2.0 ** -23   # of a power of two: bits 1 to 22 of the mantissa are set


def top_bits(x):
    return (np.ascontiguousarray(x).view(np.uint64) >> np.uint64(32)) & np.uint64(0xfffff) == 0xfffff


def block(ni, nj, nk, what):
    """Slip walls all round; `what` has the mantissas."""
    n = ni * nj * nk
    v = W.box_vertices(ni, nj, nk, 0, 0, 0, 3, spacing=1.0 / 64.0)
    rho, p = np.full(n, 1.2), np.full(n, 1.0e5)
    vx, vy, vz = np.full(n, 310.0), np.full(n, -95.0), np.full(n, 41.0)
    if what == "rho":
        rho[:] = ALMOST
    elif what == "p":
        p[:] = ALMOST * 131072.0
    elif what == "a":
        # a^2 = gamma p / rho
        p = rho * (512.0 * ALMOST) ** 2 / 1.4
    elif what == "velocity":
        vx[:], vy[:], vz[:] = 512.0 * ALMOST, -128.0 * ALMOST, 64.0 * ALMOST
    elif what == "limiter":
        # equal differences d of rho along i: the limiter's divisor 2 (64 d)^2 + 1e-12
        d = math.sqrt(0.5 * (0.125 * ALMOST - 1.0e-12)) / 64.0
        rho = 1.0 + d * np.tile(np.arange(ni), nj * nk)
    u = p / (rho * RGAS) * CV
    T = u * (1.0 / CV)
    p = rho * RGAS * T
    a = np.sqrt(1.4 * RGAS * T)
    seen = {"rho": rho, "p": p, "a": a, "velocity": np.concatenate([vx, vy, vz]),
            "limiter": 2.0 * (np.diff(rho[:ni]) * 64.0) ** 2 + 1.0e-12}[what]
    assert top_bits(seen).all()
    prim = np.stack([rho, vx, vy, vz, p, T, u, a])
    return W.BlockSpec(ni, nj, nk, v, (W.BC_SLIP_WALL,) * 6, np.zeros(8), prim)


@pytest.mark.parametrize("what", ["rho", "p", "a", "velocity", "limiter"])
@pytest.mark.parametrize("flux", ["ausmdv", "hllc", "hanel", "adaptive_hanel_ausmdv"])
@pytest.mark.parametrize("tile", [(32, 4, 3), (16, 8, 3)])
def test_fused(oracle, e4lib, what, flux, tile):
    both(oracle, [block(21, 9, 5, what)], [], flux, 2, tile)


@pytest.mark.parametrize("what", ["rho", "p", "velocity", "limiter"])
@pytest.mark.parametrize("flux", ["ausmdv", "hllc", "hanel"])
def test_general_path(oracle, e4lib, what, flux):
    b = block(21, 9, 5, what)
    b.vtx = b.vtx.copy()
    b.vtx[:, 2] *= np.where(b.vtx[:, 2] > 2.5 / 64.0, 1.25, 1.0)   # not uniform in k
    both(oracle, [b], [], flux, 2, (32, 8, 32))
