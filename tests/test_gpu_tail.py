"""The single-CTA tail: what is V vertices long is done by the whole GPU
before one CTA takes over.  Labels are whole numbers: they equal the
sequential Tarjan's."""
import numpy as np
import pytest

import detectingscc_b200 as scc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [900, 1023])
def test_word_pairs_before_the_switch(oracle_lib, k):
    """A strongly connected core, and k vertices in three-cycles in front of
    it with 20 arcs each into it: too many for the residual
    solver, few enough for the tail before any peel."""
    V, deg = 40000, 20
    rng = np.random.default_rng(k)
    i = np.arange(1, V + 1)
    o = np.arange(k)
    a = V + 1 + o
    src = np.concatenate([i, rng.integers(1, V + 1, 4 * V), a, np.repeat(a, deg)])
    dst = np.concatenate([i % V + 1, rng.integers(1, V + 1, 4 * V), np.where(o % 3 == 2, a - 2, a + 1),
                          rng.integers(1, V + 1, k * deg)])
    g = scc.graph_from_arcs(V + k, src.astype(np.int64), dst.astype(np.int64))
    lab, n = oracle_lib.tarjan(g.V, g.Fr, g.Fc)
    e = scc.Engine(0)
    try:
        e.set_tuning("trace", 4096)
        for algo in "ghxy":
            r = e.run(g, algo=algo, warp=8, force="grid")
            assert np.array_equal(r.labels, lab[1:]) and r.num_sccs == n, algo
            tail = r.stats["tail_pass"]
            assert tail > 0
            assert [p for p, _, _ in e.trace()].index("peel_init") < tail, algo
    finally:
        e.close()
