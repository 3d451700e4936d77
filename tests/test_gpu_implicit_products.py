"""The CG of the implicit solid on both sides of the rule that splits a control
point's slots over threads (100,000 points), and on point counts that fill no
CTA: the solution put into the downloaded system with plain FP64 sums.

The solver ends when ||r||^2 < eps ||r0||^2 (FP32: on the true residual of the
FP32-stored matrix), so the residual formed here is at most sqrt(eps) ||r0|| plus
the rounding of at most 375 FP64 terms (1e-12 is above it on these systems) and,
in FP32, of the double-float sums (44 bits, 1e-11).
"""
import numpy as np
import pytest

from mpm_gb300 import capi, scenes

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("grid,order", [((10, 8, 7), (1, 1, 1)), ((10, 8, 7), (2, 1, 2)), ((9, 9, 9), (2, 2, 2)),
                                        ((45, 45, 45), (1, 1, 1)), ((46, 45, 46), (1, 1, 1))])
@pytest.mark.parametrize("precision,eps", [(64, 1.0e-20), (32, 1.0e-14)])
def test_solution_satisfies_the_assembled_system(grid, order, precision, eps):
    s = scenes.cantilever(grid=grid, cell_lo=(0, 2, 2), cells=(7, 3, 3), jitter=0.1, iprop=1, idimc=order)
    s.vel[:] = np.random.default_rng(1).normal(0.0, 0.1, s.vel.shape)
    g = capi.GpuImplicitSolid(s, nr_flag=True, precision=precision)
    g.assemble()
    A, d, b = g.system()
    x, it = g.solve(eps=eps)
    g.close()
    assert it > 0
    nx, ny, nz = s.xynodec
    N = nx * ny * nz
    d, b = d.reshape(3, N), b.reshape(3, N)
    free = d > 1e-12
    for comp, nodes, _ in s.bcs:
        free[comp, nodes] = False
    xs = np.where(d > 1e-12, x.reshape(3, N) / np.where(d > 1e-12, d, 1.0), 0.0).reshape(3, nz, ny, nx)
    rx, ry, rz = order
    pad = np.pad(xs, ((0, 0), (rz, rz), (ry, ry), (rx, rx)))
    r = b * d
    r0 = np.linalg.norm(r[free])
    slot = 0
    for dz in range(2 * rz + 1):
        for dy in range(2 * ry + 1):
            for dx in range(2 * rx + 1):
                xn = pad[:, dz:dz + nz, dy:dy + ny, dx:dx + nx].reshape(3, N)
                r = r - np.einsum("rcn,cn->rn", A[slot].reshape(3, 3, N), xn)
                slot += 1
    assert np.linalg.norm(r[free]) <= (1.01 * np.sqrt(eps) + (1e-12 if precision == 64 else 1e-11)) * r0
