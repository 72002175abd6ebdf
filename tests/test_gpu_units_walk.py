"""Walks by id over the state words (32 vertices to a unit, the units dealt
out to the warps in equal rounds): vertex counts at the edges of a unit, of a
warp's 32 units and of the whole launch's.  Labels are whole numbers: they
equal the sequential Tarjan's."""
import numpy as np
import pytest

import detectingscc_b200 as scc

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def engine():
    e = scc.Engine(0)
    yield e
    e.close()


# one unit; 32 units (a warp's most); 32 warps x 32 units (one CTA's round)
@pytest.mark.parametrize("V", [1, 2, 31, 32, 33, 1023, 1024, 1025, 32767, 32768, 32769, 151552, 151553])
def test_vertex_counts(engine, oracle_lib, V):
    rng = np.random.default_rng(V)
    m = 5 * V
    # a hub reaches most vertices at once, so that the second level is found
    # bottom-up; the last id is among what is left for it
    hub = np.full(V // 2 + 1, 1)
    src = np.concatenate([rng.integers(1, V + 1, m), hub, rng.integers(1, V + 1, V // 2 + 1), [V]])
    dst = np.concatenate([rng.integers(1, V + 1, m), rng.integers(1, V + 1, V // 2 + 1), hub, [max(V - 1, 1)]])
    g = scc.graph_from_arcs(V, src.astype(np.int64), dst.astype(np.int64))
    lab, n = oracle_lib.tarjan(g.V, g.Fr, g.Fc)
    for algo in "ghxy":
        for force in ("grid", "block"):
            r = engine.run(g, algo=algo, warp=4, force=force)
            assert np.array_equal(r.labels, lab[1:]) and r.num_sccs == n, (algo, force)
