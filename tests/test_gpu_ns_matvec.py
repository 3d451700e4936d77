"""The products of the stabilized fluid's Krylov solver on both sides of the
rule that splits a node's slots over threads (32,768 nodes), and on a box whose
node count is no multiple of a CTA's 32 nodes.

The solution of mpm_ns_solve is put into the system of mpm_gpu_ns_assemble
(checked against the reference elsewhere) with plain FP64 tensor sums: on the
free rows ||b - A x|| <= 1e-9 ||b||.  The solver stops at 1e-12 ||b|| by its own
product; the sum of 432 FP64 terms adds at most 432 eps || |A| |x| ||, and
|A| |x| stays within 1e3 ||b|| on these boxes: 5e-11.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ne", [(7, 5, 4), (31, 31, 31), (32, 31, 31)])
def test_solution_satisfies_the_assembled_system(ne):
    import torch

    from mpm_gb300 import capi

    rng = np.random.default_rng(sum(ne))
    dx, nn = 0.01, np.array(ne) + 1
    N = int(np.prod(nn))
    ijk = np.stack(np.meshgrid(*[np.arange(v) for v in ne], indexing="ij"), -1).reshape(-1, 3)
    x = (ijk + 0.5 + rng.uniform(-0.3, 0.3, ijk.shape)) * dx
    k, j, i = [a.ravel() for a in np.meshgrid(*[np.arange(v) for v in nn[::-1]], indexing="ij")]
    wall = np.nonzero((i == 0) | (i == ne[0]) | (j == 0) | (j == ne[1]) | (k == 0))[0]
    top = np.nonzero(k == ne[2])[0]
    t = lambda a: torch.as_tensor(np.ascontiguousarray(a, dtype=np.float64), device="cuda:0")  # noqa: E731
    n = len(x)
    vol = np.full(n, dx ** 3)
    nvel = rng.normal(0.0, 0.01, (3, N))
    nvel[:, wall] = 0.0
    args = [t(x.T), t(1000.0 * vol), t(vol), t(nvel.ravel()), t(np.zeros(3 * N))]
    nmass = t(np.full(N, 1000.0 * dx ** 3))
    con = ((0.0,) * 3, (dx,) * 3, 1000.0, 1.0e-3, 2.0e-3, 0.25, 0.5, (0.0, 0.0, -9.8), 1.0, 1.0e-12)
    ns = capi.NsSolver(ne, *con, bcs=[(wall, np.zeros(len(wall)))] * 3 + [(top, np.zeros(len(top)))])
    (nd, npres, _, _), st = ns.solve(*args, nmass, rtol=1.0e-12)
    assert st["newton_iters"] == 1
    _, _, A, b = capi.ns_assemble(ne, *con, *args, t(np.zeros(3 * N)), t(np.zeros(N)), nmass)
    sol = torch.cat([nd, npres]).view(4, *[int(v) for v in nn[::-1]])
    pad = torch.nn.functional.pad(sol, (1, 1, 1, 1, 1, 1))
    r = b.view(4, N).clone()
    for s in range(27):
        a, c, d = s % 3, (s // 3) % 3, s // 9
        xs = pad[:, d:d + nn[2], c:c + nn[1], a:a + nn[0]].reshape(4, N)
        r -= torch.einsum("rcn,cn->rn", A[s].view(4, 4, N), xs)
    free = torch.ones(4, N, dtype=torch.bool, device="cuda:0")
    free[:3, t(wall).long()] = False
    free[3, t(top).long()] = False
    assert float(r[free].norm()) <= 1e-9 * float(b.view(4, N)[free].norm())
