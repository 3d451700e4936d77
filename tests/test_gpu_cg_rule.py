"""The CG of the implicit solid on both sides of the rule that gives p.Ap a pass of
its own (mv_dot: more than 32,768 control points).

Solution: put into the downloaded system with plain FP64 sums.  The solver ends when
||r||^2 < eps ||r0||^2 (FP32: on the true residual of the FP32-stored matrix), so the
residual formed here is at most sqrt(eps) ||r0|| plus the rounding of at most 81 FP64
terms (1e-12 is above it) and, in FP32, of the double-float sums (44 bits, 1e-11).

Launches: a solve replays its iterations from a graph or launches them one by one, in
blocks of eight either way, and mpm_stats.kernel_launches counts the same kernels.
"""
import numpy as np
import pytest

from mpm_gb300 import capi, scenes

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu
GRIDS = [(31, 31, 31), (32, 31, 31)]   # 32,768 and 33,792 control points


def solid(grid, precision, stream=None):
    s = scenes.cantilever(grid=grid, cell_lo=(0, 2, 2), cells=(12, 5, 6), jitter=0.1, iprop=1)
    s.vel[:] = np.random.default_rng(1).normal(0.0, 0.1, s.vel.shape)
    return s, capi.GpuImplicitSolid(s, nr_flag=True, precision=precision, stream=stream)


@pytest.mark.parametrize("grid", GRIDS)
@pytest.mark.parametrize("precision,eps", [(64, 1.0e-20), (32, 1.0e-14)])
def test_solution_satisfies_the_assembled_system(grid, precision, eps):
    s, g = solid(grid, precision)
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
    pad = np.pad(xs, ((0, 0), (1, 1), (1, 1), (1, 1)))
    r = b * d
    r0 = np.linalg.norm(r[free])
    for slot in range(27):
        dx, dy, dz = slot % 3, (slot // 3) % 3, slot // 9
        xn = pad[:, dz:dz + nz, dy:dy + ny, dx:dx + nx].reshape(3, N)
        r = r - np.einsum("rcn,cn->rn", A[slot].reshape(3, 3, N), xn)
    assert np.linalg.norm(r[free]) <= (1.01 * np.sqrt(eps) + (1e-12 if precision == 64 else 1e-11)) * r0


@pytest.mark.parametrize("grid", GRIDS)
def test_replayed_iterations_count_their_launches(grid):
    st = torch.cuda.Stream()
    _, g = solid(grid, 64, st.cuda_stream)
    g.assemble()
    counts = []
    for graph in (True, True, False):   # the first solve captures
        g.set_graph(graph)
        before = g.stats()["kernel_launches"]
        _, it = g.solve(eps=1.0e-20, download=False)
        counts.append((g.stats()["kernel_launches"] - before, it))
    g.close()
    assert counts[0][1] > 16
    assert counts[0] == counts[1] == counts[2], counts
