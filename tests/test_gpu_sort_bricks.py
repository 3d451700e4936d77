"""The re-sort over grids of one and of several scan segments (4096 bricks each) and
with bricks that do and do not fit the cell sort's shared memory (4096 particles).

A cell's particles come out in load order whatever the grid around the body, and
without the shifting every sum of a step is an integer sum or runs in that order: the
same body in both grids takes the same steps bit for bit, and so does a second run
(k_scatter fills the bricks in any order)."""
import numpy as np
import pytest

from mpm_gb300 import capi, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("precision", [32, 64])
@pytest.mark.parametrize("cells,npc", [((9, 5, 11), 2), ((5, 4, 9), 4), ((4, 4, 8), 5), ((1, 1, 1), 6)])
def test_the_same_body_sorts_the_same_in_any_grid(cells, npc, precision):
    runs = []
    for grid in ((20, 18, 24), (20, 18, 24), (132, 140, 72)):   # 45 and 10,395 bricks
        s = scenes.elastic_block(grid=grid, cell_lo=(3, 4, 3), cell_hi=tuple(c + o for c, o in zip(cells, (3, 4, 3))),
                                 npc=npc, fix_bottom=False, seed=4, jitter=0.2)
        s.vel[:] = np.random.default_rng(4).normal(0.0, 2.0, s.vel.shape)
        g = capi.GpuSolid(s, precision=precision, shifting=False)
        g.steps(20)   # past two re-sorts
        g.sync()
        assert g.stats()["resorts"] >= 2
        runs.append(g.particles())
        g.close()
    for k in runs[0]:
        assert np.array_equal(runs[0][k], runs[1][k]), k
        assert np.array_equal(runs[0][k], runs[2][k]), k
