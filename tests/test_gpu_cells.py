"""The per-cell scatters and the axis-by-axis gather (csrc/mpm_cells.cu) against
the staging-box kernels (mpm_config.scatter = 1), the general path of the same
calls, over precisions, shape orders and transfer schemes.

The block fills no whole brick (4 x 4 x 8 cells) in any direction and touches
the grid's walls, so every open-knot piece of the splines, partial slabs and
empty cells occur; a third of the particles have left their sorted cell since
the sort (the deferred pass), and some sit exactly on cell faces.  (FP32 linear
grids leave the faces out: there a particle on a face may count to either
cell, whose gradients differ.)

Both paths sum the same products; FP64 differs by the rounding of at most 27
terms of 64 particles (and the fixed point's 2^-44 and below): 1e-12.  FP32:
1e-5 on nodal sums, the bound of the FP32 sums against the FP64 oracle
elsewhere, and what a step makes of it on the particles.
"""
import numpy as np
import pytest

from helpers import rel_l2
from mpm_gb300 import capi, scenes

pytestmark = pytest.mark.gpu

BOUNDS = {64: dict(nodal=1e-12, x=1e-13, v=1e-12, F=1e-13, sigma=1e-10, vol=1e-13, affine=1e-9),
          32: dict(nodal=1e-5, x=1e-6, v=1e-5, F=1e-6, sigma=1e-4, vol=1e-6, affine=1e-3)}


def scene(order, scheme, cells, seed=3):
    grid = tuple(c + 2 for c in cells)
    s = scenes.elastic_block(grid=grid, cell_lo=(0, 2, 0), cell_hi=(cells[0], cells[1] + 2, cells[2]), idimc=order,
                             scheme=scheme, seed=seed, jitter=0.2)
    s.vel[:] = np.random.default_rng(seed).normal(0.0, 0.5, s.vel.shape)
    return s


@pytest.mark.parametrize("cells", [(5, 3, 9), (1, 1, 1)])
@pytest.mark.parametrize("scheme", [scenes.PIC, scenes.FLIP, scenes.TPIC, scenes.APIC])
@pytest.mark.parametrize("order", [(1, 1, 1), (2, 2, 2), (2, 1, 2)])
@pytest.mark.parametrize("precision", [64, 32])
def test_cell_scatter_matches_staging_box(precision, order, scheme, cells):
    s = scene(order, scheme, cells)
    rng = np.random.default_rng(7)
    n, dx = s.num, s.dxy[0]
    top = np.asarray(s.xyelem) * dx
    coord = s.coord.copy()
    moved = rng.random(n) < 0.34
    coord[moved] = np.clip(coord[moved] + rng.uniform(-0.9, 0.9, (int(moved.sum()), 3)) * dx, 1e-3 * dx, top - 1e-3 * dx)
    if not (precision == 32 and order == (1, 1, 1)):
        on = rng.random(n) < 0.1
        axis = rng.integers(0, 3, n)
        for d in range(3):
            q = on & (axis == d)
            coord[q, d] = dx * np.floor(coord[q, d] / dx)
    stress = rng.normal(0.0, 1.0e3, (n, 6))
    got = []
    for scatter in (0, 1):
        g = capi.GpuSolid(s, precision=precision, scatter=scatter)
        g.upload_state(coord=coord, stress=stress)
        g.p2g()
        r = {k: g.nodal(k) for k in ("nmass", "nvof", "nmome", "nforce")}
        if not (scheme == scenes.APIC and order != (1, 1, 1)):
            # APIC on a quadratic axis has no D^-1 for a particle on a wall (one of its weights is 1, the
            # others 0, and D is singular: the reference divides by zero there), and one NaN reaches every
            # particle through the fixed point's bound
            g.grid_update()
            g.g2p()
            r.update(g.particles())
            if scheme >= scenes.TPIC:
                r["affine"] = g.affine()
            g.sync()
        got.append(r)
        g.close()
    b = BOUNDS[precision]
    for k in got[0]:
        assert rel_l2(got[0][k], got[1][k]) <= b.get(k, b["nodal"]), k


@pytest.mark.parametrize("order", [(1, 1, 1), (2, 2, 2), (2, 1, 2)])
@pytest.mark.parametrize("precision", [64, 32])
def test_cell_scatter_is_reproducible_and_reports_what_left_the_grid(precision, order):
    s = scene(order, scenes.PIC, (6, 5, 10))
    runs = []
    for _ in range(2):
        g = capi.GpuSolid(s, precision=precision)
        g.steps(12)   # past a re-sort
        g.sync()
        runs.append(g.particles())
        g.close()
    for k in runs[0]:
        assert np.array_equal(runs[0][k], runs[1][k]), k
    g = capi.GpuSolid(s, precision=precision)
    coord = s.coord.copy()
    coord[5, 0] = -0.3 * s.dxy[0]
    g.upload_state(coord=coord)
    g.p2g()
    assert g.sync_status() == 4   # particle outside the grid
    g.close()


@pytest.mark.parametrize("precision", [64, 32])
def test_implicit_p2g_matches_staging_box(precision):
    s = scenes.cantilever(grid=(9, 7, 8), cells=(7, 3, 5), jitter=0.1, iprop=1)
    s.vel[:] = np.random.default_rng(2).normal(0.0, 0.1, s.vel.shape)
    out = []
    for scatter in (0, 1):
        g = capi.GpuSolid.__new__(capi.GpuImplicitSolid)
        capi.GpuSolid.__init__(g, s, precision=precision, implicit=True, scatter=scatter)
        g.radius, g.nslots = (1, 1, 1), 27
        capi._chk(g.lib.mpm_gpu_implicit_setup(g.ctx, 0, 1.0), "mpm_gpu_implicit_setup")
        g.implicit_steps(2, eps=1e-24 if precision == 64 else 1e-14)   # two: the particles carry an acceleration
        out.append(g.particles())
        g.close()
    # the solves amplify the P2G's rounding; FP32 assembles with atomics in any order
    tol = 1e-9 if precision == 64 else 1e-4
    for k in ("x", "v", "F", "sigma", "vol"):
        assert rel_l2(out[0][k], out[1][k]) <= tol, k
