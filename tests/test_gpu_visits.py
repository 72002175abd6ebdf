"""The instrumented run's vertex visits: the sweeps that read the states in id
order (half a byte a vertex) are not visits of every vertex."""
import numpy as np
import pytest

import detectingscc_b200 as scc

pytestmark = pytest.mark.gpu


# 31, 32, 33 vertices and more: the last unit of 32 ids (from 0) is full, just begun, or holds two
@pytest.mark.parametrize("leaves", [29, 30, 31, 5000])
@pytest.mark.parametrize("algo", ["g", "h"])
@pytest.mark.parametrize("force", ["grid", "block"])
def test_trimmed_vertices_are_visited_once(leaves, algo, force):
    """A pair of vertices and arcs from one of them to leaves that the degrees
    trim: every vertex is visited by the init sweep, only the pair after it
    (checked by trim-1, taken off the frontiers, listed: at most eight visits
    each)."""
    V = leaves + 2
    src = np.concatenate([[1, 2], np.full(leaves, 1)])
    dst = np.concatenate([[2, 1], np.arange(3, V + 1)])
    e = scc.Engine(0)
    try:
        r = e.run(scc.graph_from_arcs(V, src, dst), algo=algo, force=force, instrument=True)
        assert r.num_sccs == leaves + 1
        assert V <= r.stats["vertex_visits"] <= V + 16
    finally:
        e.close()
