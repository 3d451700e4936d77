"""A second load into a context that has replayed its steps from a graph: the graph
holds the buffers, the count and the largest mass of the first load, and what the
allocator returns for the second may lie at the same addresses.

The steps after it equal a fresh context's bit for bit (both start with a sort, on an
even step).
"""
import numpy as np
import pytest

from mpm_gb300 import capi, scenes

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("cells", [(6, 5, 9), (5, 5, 8)])
@pytest.mark.parametrize("precision", [32, 64])
def test_steps_after_a_second_load_match_a_fresh_context(precision, cells):
    st = torch.cuda.Stream()
    first = scenes.elastic_block(grid=(16, 15, 20), cell_lo=(3, 4, 3), cell_hi=(9, 9, 12), fix_bottom=False)
    second = scenes.elastic_block(grid=(16, 15, 20), cell_lo=(3, 4, 3), cell_hi=tuple(c + o for c, o in zip(cells, (3, 4, 3))),
                                  fix_bottom=False, rho=1.0e9, seed=5)
    for i, s in enumerate((first, second)):
        s.vel[:] = np.random.default_rng(i).normal(0.0, 0.3, s.vel.shape)
    out = []
    for again in (True, False):
        g = capi.GpuSolid(first if again else second, precision=precision, stream=st.cuda_stream)
        if again:
            g.steps(64)
            g.load(second.coord, second.vel, second.mass, second.vol0, matid=second.matid)
        g.steps(64)
        g.sync()
        out.append(g.particles())
        g.close()
    for k in out[0]:
        assert np.array_equal(out[0][k], out[1][k]), k
