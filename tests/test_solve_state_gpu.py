"""What a solve and a host-driven push leave behind, and what engines and
streams share."""
import numpy as np
import pytest

from test_long_lists_gpu import edged_graph
from test_passes_gpu import EPS, engine

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
if not torch.cuda.is_available():
    pytest.skip("needs a GPU", allow_module_level=True)


@pytest.mark.parametrize("sweep", [False, True])
@pytest.mark.parametrize("n,cap", [(2500, 900), (2500, 1), (70001, 20000), (300007, 10 ** 9)])
def test_pending_lists_after_a_solve(n, cap, sweep):
    """The pending list of every chunk is that of the last snapshot, whichever pass it ended: the
    vertices whose residual is above eps, none of them after convergence."""
    idx, adj = edged_graph(n, 4, symmetric=True)
    eng = engine(n, idx, adj, "pr", cap)
    assert (eng.nc == 1) == (cap > len(adj))
    eng.set_chunk_sweep(sweep)
    eng.set_sweep_demand(0.2)
    ends = np.append(eng.chunk_v0[1:], n)
    few = range(eng.nc) if eng.nc < 50 else list(range(20)) + list(range(eng.nc - 20, eng.nc))
    for passes in (0, 1, 2, 3, 4, 9, 10, 100000):
        eng.solve(max_passes=passes)
        pending = np.abs(eng.read(0, residual=True)) > np.float32(EPS)
        assert pending.any() == (passes < 100000)
        for c in few:
            lo, hi = int(eng.chunk_v0[c]), int(ends[c])
            assert np.array_equal(np.sort(eng.chunk_list(c)), lo + np.nonzero(pending[lo:hi])[0]), (passes, c)
    eng.close()
