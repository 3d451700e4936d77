"""The FLIP gather of the FP32 linear path, whose bricks bring their particles' old
velocities into shared memory 4096 at a time, against the staging-box kernels
(mpm_config.scatter = 1): bricks below, at and above one chunk, ragged cells, and
particles that have left their sorted cell.

Both paths sum the same products in FP32; the bounds are those of the FP32 cell
scatters against the same kernels: 1e-5 on velocities and nodal sums, 1e-6 on
positions.
"""
import numpy as np
import pytest

from helpers import rel_l2
from mpm_gb300 import capi, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("moved", [0.0, 0.2])
@pytest.mark.parametrize("cells,npc", [((5, 3, 9), 2), ((4, 4, 8), 3), ((6, 5, 10), 4), ((4, 4, 4), 4), ((1, 2, 1), 5)])
def test_flip_velocities_match_staging_box(cells, npc, moved):
    s = scenes.elastic_block(grid=tuple(c + 2 for c in cells), cell_lo=(0, 2, 0),
                             cell_hi=(cells[0], cells[1] + 2, cells[2]), npc=npc, scheme=scenes.FLIP, seed=4,
                             jitter=0.2)
    rng = np.random.default_rng(5)
    s.vel[:] = rng.normal(0.0, 0.5, s.vel.shape)
    n, dx = s.num, s.dxy[0]
    coord = s.coord.copy()
    out = rng.random(n) < moved
    coord[out] += rng.uniform(-0.9, 0.9, (int(out.sum()), 3)) * dx
    q = np.clip(coord, 1e-3 * dx, np.asarray(s.xyelem) * dx - 1e-3 * dx) / dx
    coord = (np.floor(q) + np.clip(q - np.floor(q), 1e-3, 0.999)) * dx   # FP32: off the cell faces
    stress = rng.normal(0.0, 1.0e3, (n, 6))
    got = []
    for scatter in (0, 1):
        g = capi.GpuSolid(s, precision=32, scatter=scatter)
        g.upload_state(coord=coord, stress=stress)
        g.p2g()
        g.grid_update()
        g.g2p()
        got.append(g.particles())
        g.close()
    assert rel_l2(got[0]["v"], got[1]["v"]) <= 1e-5
    assert rel_l2(got[0]["x"], got[1]["x"]) <= 1e-6
