"""Who derives the fixed-point scales of a step and sums the shifting's nei^2: the
P2G, the first gather, the affine re-projection and the F-bar projection each
derive theirs in every CTA, the first grid pass leaves one partial per CTA and the
second adds them.  The same body in a grid whose tiles have a CTA each and in one
whose tiles are listed: the nodal sums are the same integers, and only the order of
the FP64 sum of nei^2 differs (its rounding, 1e-13 at 10,000 terms, reaches the
positions through the shifting): 1e-12 in FP64; in FP32 a position may round the
other way, 1e-6 (stress, a difference of positions over 1 / dt: 1e-4)."""
import numpy as np
import pytest

from helpers import rel_l2
from mpm_gb300 import capi, scenes

pytestmark = pytest.mark.gpu

BOUNDS = {64: dict(x=1e-12, v=1e-12, F=1e-12, sigma=1e-11, vol=1e-12),
          32: dict(x=1e-6, v=1e-5, F=1e-6, sigma=1e-4, vol=1e-6)}


@pytest.mark.parametrize("fbar", [False, True])
@pytest.mark.parametrize("scheme", [scenes.PIC, scenes.FLIP, scenes.TPIC, scenes.APIC])
@pytest.mark.parametrize("order", [(1, 1, 1), (2, 2, 2)])
@pytest.mark.parametrize("precision", [64, 32])
def test_direct_and_listed_tiles_take_the_same_steps(precision, order, scheme, fbar):
    out = []
    for grid in ((16, 14, 17), (90, 80, 70)):   # 12 and 1,188 tiles
        s = scenes.elastic_block(grid=grid, cell_lo=(3, 4, 3), cell_hi=(11, 9, 12), scheme=scheme, idimc=order,
                                 fix_bottom=False, seed=4, jitter=0.2)
        # crowded nodes: the shifting has something to do
        s.vol0[:] *= 1.3
        s.vel[:] = np.random.default_rng(4).normal(0.0, 0.5, s.vel.shape)
        g = capi.GpuSolid(s, precision=precision, shifting=True, fbar=fbar)
        g.steps(10)   # past a re-sort
        g.sync()
        out.append(g.particles())
        g.close()
    for k, b in BOUNDS[precision].items():
        assert rel_l2(out[0][k], out[1][k]) <= b, k
