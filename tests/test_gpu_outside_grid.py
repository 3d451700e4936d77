"""A particle outside the grid (reported as an error by the next mpm_gpu_sync) moves
with the weights of the nearest cell as axis_eval gives them, in its scatter, its
gather and its update alike: inside the grid the FP64 gathers take a shorter way.

The gathered velocity is compared with the staging-box route's (mpm_config.scatter =
1), the new position of linear grids with dt sum N v over the downloaded nodal
velocities, N = product of 1 - |x - x_i| / dx; both sum the same eight to 27 terms:
1e-12.
"""
import numpy as np
import pytest

from helpers import rel_l2
from mpm_gb300 import capi, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("scheme", [scenes.PIC, scenes.FLIP])
@pytest.mark.parametrize("order", [(1, 1, 1), (2, 2, 2), (2, 1, 2)])
def test_particles_outside_the_grid_keep_their_weights(order, scheme):
    s = scenes.elastic_block(grid=(7, 6, 9), cell_lo=(0, 0, 0), cell_hi=(7, 6, 9), idimc=order, scheme=scheme,
                             fix_bottom=False)
    rng, dx = np.random.default_rng(2), s.dxy[0]
    s.vel[:] = rng.normal(0.0, 0.5, s.vel.shape)
    top = np.asarray(s.xyelem) * dx
    coord = s.coord.copy()
    out = rng.choice(s.num, 60, replace=False)
    for i, p in enumerate(out):
        d = i % 3
        coord[p, d] = -rng.uniform(0.05, 0.45) * dx if i % 2 else top[d] + rng.uniform(0.05, 0.45) * dx
    got = []
    for scatter in (0, 1):
        g = capi.GpuSolid(s, precision=64, scatter=scatter, shifting=False)
        g.upload_state(coord=coord)
        g.p2g()
        g.grid_update()
        g.g2p()
        assert g.sync_status() == 4
        got.append(dict(g.particles(), nvel=g.nodal("nvel")))
        g.close()
    assert np.isfinite(got[0]["x"]).all()
    assert rel_l2(got[0]["v"][out], got[1]["v"][out]) <= 1e-12
    assert rel_l2(got[0]["x"][out], got[1]["x"][out]) <= 1e-12
    if order != (1, 1, 1):
        return
    cell = np.clip(np.floor(coord[out] / dx).astype(int), 0, np.asarray(s.xyelem) - 1)
    nx, ny, _ = s.xynodec
    move = np.zeros((len(out), 3))
    for k in range(8):
        n = cell + [k & 1, k >> 1 & 1, k >> 2]
        w = np.prod(1.0 - np.abs(coord[out] - n * dx) / dx, axis=1)
        move += w[:, None] * got[0]["nvel"][:, n[:, 0] + nx * (n[:, 1] + ny * n[:, 2])].T
    assert rel_l2(got[0]["x"][out], coord[out] + s.dt * move) <= 1e-12
