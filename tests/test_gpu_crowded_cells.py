"""Crowded cells in the per-cell scatters (csrc/mpm_cells.cu): bricks whose fullest
cell holds more than about 32 particles are cut into shares.

Sums: against the staging-box kernels (mpm_config.scatter = 1) for cells of 1 to 600
particles on both sides of the rule, next to one another, a third of the particles
outside their sorted cell; the same bounds as between these routes elsewhere (both
sum the same products: FP64 to 1e-12, FP32 to 1e-5 on nodal sums), and the same
bits from run to run although the shares are listed in any order.

Time: the staging box spreads a brick's particles over as many CTAs as they fill,
so a few bricks of 216 particles per cell showed cells that are walked one particle
after another (APIC in FP64: 1718 against 826 us for P2G and re-projection at 27,000
particles; 313 with the shares).  The shares have to be the faster route there.
"""
import numpy as np
import pytest

from helpers import rel_l2
from mpm_gb300 import capi, scenes

pytestmark = pytest.mark.gpu


def uneven(order, scheme, counts, seed=3):
    """A row of cells along x (and a second one in another brick) with the given particle counts."""
    s = scenes.elastic_block(grid=(len(counts) + 2, 9, 10), cell_lo=(1, 1, 1), cell_hi=(2, 2, 2), npc=1, idimc=order,
                             scheme=scheme, fix_bottom=False)
    rng, dx = np.random.default_rng(seed), s.dxy[0]
    cell = np.concatenate([np.tile([i + 1, row, row], (n, 1)) for row in (2, 7) for i, n in enumerate(counts)])
    n = len(cell)
    order_ = rng.permutation(n)   # load order is not cell order
    x = (cell + rng.uniform(0.02, 0.98, (n, 3)))[order_] * dx
    vp = dx ** 3 / 8
    return scenes.Scene(**{**s.__dict__, "coord": x, "vel": rng.normal(0.0, 0.5, (n, 3)), "mass": np.full(n, 1000.0 * vp),
                           "vol0": np.full(n, vp), "matid": np.zeros(n, dtype=np.int32)})


@pytest.mark.parametrize("counts", [(47, 48, 1, 49), (8, 600, 0, 31, 79, 80)])
@pytest.mark.parametrize("scheme", [scenes.PIC, scenes.APIC])
@pytest.mark.parametrize("precision,order", [(64, (1, 1, 1)), (64, (2, 2, 2)), (32, (2, 2, 2)), (32, (2, 1, 2))])
def test_shares_match_the_staging_box(precision, order, scheme, counts):
    s = uneven(order, scheme, counts)
    rng, dx = np.random.default_rng(9), s.dxy[0]
    coord = s.coord.copy()
    moved = rng.random(s.num) < 0.34
    coord[moved] += rng.uniform(-0.9, 0.9, (int(moved.sum()), 3)) * dx
    stress = rng.normal(0.0, 1.0e3, (s.num, 6))
    got = []
    for scatter in (0, 1, 0):
        g = capi.GpuSolid(s, precision=precision, scatter=scatter)
        g.upload_state(coord=coord, stress=stress)
        g.p2g()
        r = {k: g.nodal(k) for k in ("nmass", "nvof", "nmome", "nforce")}
        g.grid_update()
        g.g2p()
        r["nvel"] = g.nodal("nvel")
        g.sync()
        got.append(r)
        g.close()
    for k in got[0]:
        assert rel_l2(got[0][k], got[1][k]) <= (1e-12 if precision == 64 else 1e-5), k
        assert np.array_equal(got[0][k], got[2][k]), k


def test_crowded_cells_are_not_slower_than_in_the_staging_box():
    s = scenes.elastic_block(grid=(13, 13, 13), cell_lo=(4, 4, 4), cell_hi=(9, 9, 9), npc=6, scheme=scenes.APIC,
                             fix_bottom=False, jitter=0.05, dt=1e-7)
    took = []
    for scatter in (0, 1):
        g = capi.GpuSolid(s, precision=64, scatter=scatter)
        g.steps(8)
        g.enable_kernel_timing(True)
        best = np.inf
        for _ in range(5):
            g.kernel_times()
            g.steps(4)
            t = g.kernel_times()
            best = min(best, t["p2g"][0] + t["g2p_musl"][0])
        took.append(best)
        g.close()
    assert took[0] <= took[1], took
