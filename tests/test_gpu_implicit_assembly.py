"""The cell-wise assembly of the FP32 implicit operator (isotropic materials)
against the atomic one of the same context (mpm_config.scatter = 1), and both
against the FP64 operator.

The block fills no whole brick, its cells hold 8 or 64 particles (less and more
than one round of a CTA's shared memory), a third of the particles have left
their sorted cell, and F and the stress are those of a deformed body.

Tolerance: both sum the same FP32 products.  A block of the matrix has at most 64 x 8
particle terms of either sign; in the 2-norm over the matrix their rounding stays below
sqrt(512) 2^-24 = 1.4e-6 of the terms, and a particle's own terms (coordinate,
shape functions, F, stress: about ten roundings, the coordinate's divided by the
cell) below 4e-6.  1e-5 for the scaled matrix, 1e-5 for D^-1/2 and the RHS.  The
cell-wise sums are rounded no more often than the atomic ones: their error
against FP64 may not exceed the atomic one's by more than a tenth (plus 2^-24).
"""
import numpy as np
import pytest

from helpers import rel_l2
from mpm_gb300 import capi, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells,npc", [((7, 3, 9), 2), ((2, 5, 3), 4), ((1, 1, 1), 2)])
@pytest.mark.parametrize("iprop,nr", [(-1, False), (0, True), (1, True), (1, False)])
@pytest.mark.parametrize("order", [(1, 1, 1), (2, 2, 2), (2, 1, 2)])
def test_cell_assembly_matches_atomics(order, iprop, nr, cells, npc):
    s = scenes.cantilever(grid=tuple(c + 3 for c in cells), cell_lo=(0, 1, 2), cells=cells, npc=npc, jitter=0.2,
                          iprop=iprop, idimc=order)
    rng = np.random.default_rng(11)
    n, dx = s.num, s.dxy[0]
    s.vel[:] = rng.normal(0.0, 0.1, s.vel.shape)
    coord = s.coord.copy()
    moved = rng.random(n) < 0.34
    top = np.asarray(s.xyelem) * dx
    coord[moved] = np.clip(coord[moved] + rng.uniform(-0.9, 0.9, (int(moved.sum()), 3)) * dx, 1e-2 * dx, top - 1e-2 * dx)
    # FP32 coordinates can land on the other side of a face: keep off the faces
    q = coord / dx
    coord = (np.floor(q) + np.clip(q - np.floor(q), 1e-2, 0.99)) * dx
    F = np.eye(3).reshape(1, 9) + rng.normal(0.0, 0.03, (n, 9))
    stress = rng.normal(0.0, 2.0e5, (n, 6))
    out = {}
    for key, precision, scatter in (("ref", 64, 1), ("atomic", 32, 1), ("cells", 32, 0)):
        g = capi.GpuSolid.__new__(capi.GpuImplicitSolid)
        capi.GpuSolid.__init__(g, s, precision=precision, implicit=True, scatter=scatter)
        g.radius, g.nslots = order, int(np.prod([2 * r + 1 for r in order]))
        capi._chk(g.lib.mpm_gpu_implicit_setup(g.ctx, int(nr), 1.0), "mpm_gpu_implicit_setup")
        g.upload_state(coord=coord, F=F, stress=stress)
        g.assemble()
        out[key] = dict(zip(("A", "d", "b"), g.system()))
        g.close()
    for k in ("A", "d", "b"):
        err = {w: rel_l2(out[w][k], out["ref"][k]) for w in ("atomic", "cells")}
        assert rel_l2(out["cells"][k], out["atomic"][k]) <= 1e-5, (k, err)
        assert err["cells"] <= 1.1 * err["atomic"] + 2.0 ** -24, (k, err)
