"""A drop-in solve that fails leaves zeros in `dist`, not an earlier solve's
distances (predecessors: -1)."""
import numpy as np
import pytest

from fastapsp_b200 import FapError, fapGraph
from fastapsp_b200 import generators as G

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("paths", [False, True])
def test_failed_solve_leaves_no_stale_distances(cuda_ok, paths):
    el = G.grid_graph(20, 21, wmin=1, wmax=9, seed=5)
    ro, col, w = G.edges_to_csr(el)
    g = fapGraph.from_csr(el.n, int(ro[-1]), ro, col, w, 4, directed=el.directed)
    g.preCondition()
    g.solve(paths)
    first = np.array(g.getAllDistance())
    assert first.max() > 0
    g.setMaxResidentRows(1)                    # no part fits
    with pytest.raises(FapError):
        g.solve(paths)
    assert not np.asarray(g.getAllDistance()).any()
    if paths:
        assert (np.asarray(g.getAllPath()) == -1).all()
    g.setMaxResidentRows(0)
    g.solve(paths)
    assert np.array_equal(np.array(g.getAllDistance()), first)
