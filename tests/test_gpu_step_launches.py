"""The FP32 linear step's shorter launch sequence: the moment kernels take the
particles that left their sorted cell from their brick's own queue, the P2G
starts the step itself, and a grid of few tiles runs its grid passes without a
tile list.

The particles are compared with the corner-form kernels (mpm_gpu_set_tuning 2,
3, 3), which queue them for launches of their own; both forms differ by FP32
rounding, bounded as in the explicit tests: x 1e-6, v 1e-5, F and vol 1e-6,
stress 1e-4 of its norm.  Direct and listed tiles add the same fixed-point sums
and differ in the order of one FP64 sum (the shifting's), below FP32: 1e-6.
"""
import numpy as np
import pytest

from helpers import rel_l2
from mpm_gb300 import capi, scenes

pytestmark = pytest.mark.gpu
BOUNDS = dict(x=1e-6, v=1e-5, F=1e-6, sigma=1e-4, vol=1e-6)


def block(scheme=scenes.PIC, grid=(13, 12, 16), model=0):
    s = scenes.elastic_block(grid=grid, cell_lo=(2, 3, 2), cell_hi=(11, 9, 12), scheme=scheme, fix_bottom=False,
                             iprop=model, seed=4)
    s.vel[:] = np.random.default_rng(4).normal(0.0, 0.5, s.vel.shape)
    return s


@pytest.mark.parametrize("share", [0.0, 0.01, 0.3, 1.0])
@pytest.mark.parametrize("scheme", [scenes.PIC, scenes.FLIP])
def test_particles_outside_their_cell_match_the_corner_form(scheme, share):
    s = block(scheme)
    rng = np.random.default_rng(1)
    coord = s.coord.copy()
    m = rng.random(s.num) < share
    coord[m] += rng.choice([-1.3, -0.8, 0.8, 1.3], (int(m.sum()), 3)) * s.dxy[0]
    stress = rng.normal(0.0, 1e3, (s.num, 6))
    out = []
    for tune in (None, (2, 3, 3)):
        g = capi.GpuSolid(s, precision=32)
        if tune:
            g.set_tuning(*tune)
        g.upload_state(coord=coord, stress=stress)
        g.steps(2)
        g.sync()
        if share > 0.0:
            assert g.stats()["tile_misses"] > 0
        out.append(g.particles())
        g.close()
    for k, b in BOUNDS.items():
        assert rel_l2(out[0][k], out[1][k]) <= b, k


def test_moment_kernels_report_a_particle_outside_the_grid():
    s = block()
    g = capi.GpuSolid(s, precision=32)
    coord = s.coord.copy()
    coord[17, 2] = -0.4 * s.dxy[0]
    g.upload_state(coord=coord)
    g.steps(1)
    assert g.sync_status() == 4
    g.close()


def test_steps_after_uploads_and_load_changes_match_a_fresh_context():
    """The P2G of each step derives its scales from the bounds that the step before, an upload or a new load left."""
    s = block()
    g = capi.GpuSolid(s, precision=32)
    g.steps(3)
    g.upload_state(coord=s.coord, vel=100.0 * s.vel, F=np.tile(np.eye(3).ravel(), (s.num, 1)),
                   stress=np.zeros((s.num, 6)), vol=s.vol0)
    g.steps(2, facl=3.0)
    g.p2g(3.0)
    m = g.nodal("nmass").sum()
    g.sync()
    s.vel *= 100.0
    f = capi.GpuSolid(s, precision=32)
    f.steps(2, facl=3.0)
    f.sync()
    a, b = g.particles(), f.particles()
    for k, t in BOUNDS.items():   # the two contexts sort at different steps: FP32 rounding
        assert rel_l2(a[k], b[k]) <= t, k
    assert abs(m - s.mass.sum()) <= 1e-5 * s.mass.sum()
    g.close()
    f.close()


@pytest.mark.parametrize("model", [0, 1])
def test_direct_tiles_match_the_tile_list(model):
    out = []
    for grid in ((13, 12, 16), (80, 80, 80)):   # 12 tiles and 1,331
        g = capi.GpuSolid(block(grid=grid, model=model), precision=32)
        g.steps(20)
        g.sync()
        out.append(g.particles())
        g.close()
    for k in BOUNDS:
        assert rel_l2(out[0][k], out[1][k]) <= 1e-6, k
