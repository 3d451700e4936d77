"""The flexible GCR passes with every window of kept directions (both widths of
their loops), on grids whose vectors are and are not a multiple of four values
long and fill no block: the solution put into the downloaded system with plain
FP64 sums.

The solver ends on the true residual, ||r||^2 < eps ||r0||^2, so the residual formed
here is at most sqrt(eps) ||r0|| plus the rounding of at most 81 FP64 terms (1e-12
is above it) and, in FP32, of the double-float sums (44 bits, 1e-11).
"""
import numpy as np
import pytest

from mpm_gb300 import capi, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("window", [1, 2, 4, 8])
@pytest.mark.parametrize("grid", [(10, 8, 7), (9, 9, 9), (13, 6, 7), (24, 20, 21)])
@pytest.mark.parametrize("precision,eps", [(64, 1.0e-18), (32, 1.0e-14)])
def test_learned_solution_satisfies_the_assembled_system(monkeypatch, grid, window, precision, eps):
    from mpm_gb300 import train_precond

    params = train_precond.load_weights()
    if params is None:
        pytest.skip("no committed preconditioner parameters")
    monkeypatch.setenv("MPM_GB300_GCR_WINDOW", str(window))
    s = scenes.cantilever(grid=grid, cell_lo=(0, 2, 2), cells=tuple(n - 3 for n in grid), jitter=0.1, iprop=1)
    s.vel[:] = np.random.default_rng(1).normal(0.0, 0.1, s.vel.shape)
    g = capi.GpuImplicitSolid(s, nr_flag=True, precision=precision)
    net = capi.PrecondNet(s.xynodec)
    net.set_params(params)
    g.set_precond(net)
    g.assemble()
    A, d, b = g.system()
    x, it = g.solve(eps=eps)
    g.set_precond(None)
    g.close()
    assert it > 0
    nx, ny, nz = s.xynodec
    N = nx * ny * nz
    d, b = d.reshape(3, N), b.reshape(3, N)
    free = d > 1e-12
    for comp, nodes, _ in s.bcs:
        free[comp, nodes] = False
    xs = np.where(d > 1e-12, x.reshape(3, N) / np.where(d > 1e-12, d, 1.0), 0.0).reshape(3, nz, ny, nx)
    pad = np.pad(xs, ((0, 0), (1, 1), (1, 1), (1, 1)))
    r = b * d
    r0 = np.linalg.norm(r[free])
    for slot in range(27):
        dx, dy, dz = slot % 3, (slot // 3) % 3, slot // 9
        xn = pad[:, dz:dz + nz, dy:dy + ny, dx:dx + nx].reshape(3, N)
        r = r - np.einsum("rcn,cn->rn", A[slot].reshape(3, 3, N), xn)
    assert np.linalg.norm(r[free]) <= (1.01 * np.sqrt(eps) + (1e-12 if precision == 64 else 1e-11)) * r0
