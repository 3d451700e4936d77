"""MPM_GB300_PDL=0 turns programmatic dependent launch off in every kernel launch of
the library, so that the switch tells an ordering fault from another one: on the
sources (every launch() takes its flag from the switch), and on a GPU the implicit
solvers and the fluid step run to the same results without it.

Results: the solves end below the given residual either way, and their assemblies add
FP64 numbers with atomics in any order: 1e-9, as between two runs elsewhere.
"""
import glob
import os
import re

import numpy as np
import pytest

from helpers import rel_l2
from mpm_gb300 import build, capi, scenes


def test_every_launch_takes_the_switch():
    flags, lets = set(), set()
    for path in glob.glob(os.path.join(build.CSRC, "*.cu*")):
        text = re.sub(r"//.*", "", open(path).read())
        flags |= {m.strip() for m in re.findall(r"(?<![\w.>])launch\(([^,()]+),", text) if not m.startswith("bool ")}
        lets |= set(re.findall(r"bool pdl = ([^;)]+);", text))
    assert flags and all("pdl" in f for f in flags), flags
    assert lets and all("pdl" in v for v in lets), lets


def implicit(precision, learned):
    s = scenes.cantilever(grid=(10, 8, 7), cell_lo=(0, 2, 2), cells=(7, 3, 3), jitter=0.1, iprop=1)
    s.vel[:] = np.random.default_rng(1).normal(0.0, 0.1, s.vel.shape)
    g = capi.GpuImplicitSolid(s, nr_flag=True, precision=precision)
    if learned:
        from mpm_gb300 import train_precond

        params = train_precond.load_weights()
        if params is None:
            pytest.skip("no committed preconditioner parameters")
        net = capi.PrecondNet(s.xynodec)
        net.set_params(params)
        g.set_precond(net)
    g.implicit_steps(2, eps=1e-24 if precision == 64 else 1e-14)
    p = g.particles()
    g.sync()
    g.set_precond(None)
    g.close()
    return p


def fluid():
    import torch

    ne, dx = np.array([5, 4, 6]), 0.01
    rng = np.random.default_rng(3)
    ijk = np.stack(np.meshgrid(*[np.arange(2 * v) for v in ne], indexing="ij"), -1).reshape(-1, 3)
    x = (ijk + 0.5 + rng.uniform(-0.1, 0.1, ijk.shape)) * (dx / 2)
    nn = ne + 1
    k, j, i = (a.ravel() for a in np.meshgrid(*[np.arange(n) for n in nn[::-1]], indexing="ij"))
    wall = np.nonzero((i == 0) | (i == ne[0]) | (j == 0) | (j == ne[1]) | (k == 0))[0]
    top = np.nonzero(k == ne[2])[0]
    bcs = [(wall, np.zeros(len(wall)))] * 3 + [(top, np.zeros(len(top)))]
    ns = capi.NsSolver(ne, (0.0,) * 3, (dx,) * 3, 1000.0, 1.0e-3, 2.0e-3, 0.25, 0.5, (0.0, 0.0, -9.8), 1.0, 1.0e-12,
                       bcs=bcs)
    n = len(x)
    vol = torch.full((n,), dx ** 3 / 8, dtype=torch.float64, device="cuda")
    xs = torch.as_tensor(np.ascontiguousarray(x.T)).cuda()
    v = torch.as_tensor(rng.normal(0.0, 0.02, (3, n))).cuda()
    a, p = torch.zeros(3, n, dtype=torch.float64, device="cuda"), torch.zeros(n, dtype=torch.float64, device="cuda")
    ns.step(xs, v, a, p, 1000.0 * vol, vol, scheme=scenes.FLIP, rtol=1.0e-12)
    torch.cuda.synchronize()
    return {"x": xs.cpu().numpy(), "v": v.cpu().numpy()}


@pytest.mark.gpu
@pytest.mark.parametrize("what,tol", [(lambda: implicit(64, False), 1e-9), (lambda: implicit(32, False), 1e-4),
                                      (lambda: implicit(32, True), 1e-4), (fluid, 1e-9)],
                         ids=["cg64", "cg32", "gcr32", "fluid"])
def test_solvers_without_programmatic_launch(monkeypatch, what, tol):
    out = []
    for v in ("1", "0"):
        monkeypatch.setenv("MPM_GB300_PDL", v)
        out.append(what())
    for k in ("x", "v"):
        assert rel_l2(out[1][k], out[0][k]) <= tol, k
