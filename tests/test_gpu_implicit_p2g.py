"""The implicit solid's P2G (the particles' accelerations among its sums) against
the oracle's, sum by sum, with particles that have left their sorted cell.

The particles sit on a lattice of 2^-16 in cells of 2^-6, at odd multiples, with
masses and volumes that are powers of two: positions, offsets and shape functions
are exact in FP32, and a contribution's only roundings are those of its products.
The particles' accelerations are those of a step from rest under a random
stress, with gamma = 1/2 and dt = 2^-10: v = gamma dt a exactly, so that the downloaded
velocities give them to the last bit.  The oracle's momentum sums of a scene that
moves with v, a and |a| are the references (FP64).

FP32, u = 2^-24, S = sum N m |a|: a linear contribution's weight is rounded once (three
factors of at most 11 bits), a quadratic one's twice (factors of 21 bits), the
product with a velocity once more, the downloaded sum once.  The sums themselves
are exact to 48 bits: |error| <= (k + 1) u S with k = 1, 2 for mass and volume and one
more for momentum and N m a.  (Plain FP32 sums of 64 particles leave these bounds.)
FP64: at most 216 x 27 terms, 1e-12 S, and the fixed point's last place, 1e-12 of the
largest sum.
"""
import numpy as np
import pytest

from mpm_gb300 import capi, scenes
from oracle import port

pytestmark = pytest.mark.gpu
DX, DT = 2.0 ** -6, 2.0 ** -10


def lattice(x, top):
    q = 2 * np.floor(np.clip(x, 2.0 ** -15, top - 2.0 ** -15) * 2.0 ** 15) + 1
    return q * 2.0 ** -16


def oracle_sums(s, coord, vel):
    t = scenes.Scene(**{**s.__dict__, "coord": coord, "vel": np.ascontiguousarray(vel)})
    o = port.PortSolid(t)
    o.p2g()
    return o.nodal("nmass"), o.nodal("nvof"), o.nodal("nmome")


@pytest.mark.parametrize("scatter", [0, 1])
@pytest.mark.parametrize("npc", [2, 4])
@pytest.mark.parametrize("order", [(1, 1, 1), (2, 2, 2), (2, 1, 2)])
@pytest.mark.parametrize("precision", [64, 32])
def test_sums_match_the_oracle(precision, order, npc, scatter):
    cells = (6, 3, 5)
    s = scenes.cantilever(grid=(9, 6, 8), dx=DX, cells=cells, npc=npc, jitter=0.1, rho=1024.0, iprop=1, idimc=order,
                          scheme=scenes.FLIP, dt=DT)
    rng = np.random.default_rng(5)
    n, top = s.num, np.asarray(s.xyelem) * DX
    s.coord[:] = lattice(s.coord, top)
    g = capi.GpuSolid.__new__(capi.GpuImplicitSolid)
    capi.GpuSolid.__init__(g, s, precision=precision, implicit=True, scatter=scatter)
    g.radius, g.nslots = order, int(np.prod([2 * r + 1 for r in order]))
    capi._chk(g.lib.mpm_gpu_implicit_setup(g.ctx, 1, 1.0), "mpm_gpu_implicit_setup")
    g.upload_state(stress=rng.normal(0.0, 1.0e4, (n, 6)))
    g.implicit_steps(1, eps=1e-24 if precision == 64 else 1e-14)
    acc = g.particles()["v"] / (0.5 * DT)
    coord = s.coord.copy()
    moved = rng.random(n) < 0.34
    coord[moved] = lattice(coord[moved] + rng.uniform(-0.9, 0.9, (int(moved.sum()), 3)) * DX, top)
    vel = np.abs(rng.normal(1.0, 0.3, (n, 3))).astype(np.float32).astype(np.float64)
    g.upload_state(coord=coord, vel=vel, vol=s.vol0)
    g.assemble()
    got = {k: g.nodal(k) for k in ("nmass", "nvof", "nmome", "nforce")}
    g.sync()
    g.close()
    assert np.abs(acc).min() > 0.0
    mass, nvof, mome = oracle_sums(s, coord, vel)
    force, size = oracle_sums(s, coord, acc)[2], oracle_sums(s, coord, np.abs(acc))[2]
    k = 1 if order == (1, 1, 1) else 2
    u = 2.0 ** -24
    for name, ref, scale, rounds in (("nmass", mass, mass, k + 1), ("nvof", nvof, nvof, k + 1),
                                     ("nmome", mome, mome, k + 2), ("nforce", force, size, k + 2)):
        rel = 1e-12 if precision == 64 else 1.0001 * rounds * u
        slack = 1e-12 * scale.max() + (s.mtol if name == "nvof" else 0.0)
        worst = float(np.max((np.abs(got[name] - ref) - slack) / np.maximum(scale, 1e-300)))
        assert worst <= rel, (name, worst / u)
