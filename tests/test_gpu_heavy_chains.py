"""Long chains of vertices whose lists are cut into chunks (above 256 arcs):
each hop can take two passes, one that cuts the list and one that walks it,
and such a run still has to end with the right labels.  Labels are whole
numbers: they equal the sequential Tarjan's."""
import numpy as np
import pytest

import detectingscc_b200 as scc

pytestmark = pytest.mark.gpu


def _cycle(n, mult, star, rev):
    """A cycle of n vertices (their ids along the way), every arc mult times,
    and a two-way star, which takes the first pivot when it has the larger
    degrees."""
    c = np.arange(1, n + 1)
    src, dst = np.repeat(c, mult), np.repeat(c % n + 1, mult)
    if rev:
        src, dst = dst, src
    s0, leaf = n + 1, np.arange(n + 2, n + 2 + star)
    src = np.concatenate([src, np.full(star, s0), leaf])
    dst = np.concatenate([dst, leaf, np.full(star, s0)])
    return scc.graph_from_arcs(n + 1 + star, src.astype(np.int64), dst.astype(np.int64))


@pytest.fixture(scope="module")
def engine():
    e = scc.Engine(0)
    yield e
    e.close()


@pytest.mark.parametrize("rev", [False, True])
@pytest.mark.parametrize("star", [0, 600])   # the search from the pivot walks the cycle; the peels do
@pytest.mark.parametrize("mult", [256, 257, 513])
def test_two_passes_a_hop(engine, oracle_lib, mult, star, rev):
    g = _cycle(1500, mult, star, rev)
    lab, n = oracle_lib.tarjan(g.V, g.Fr, g.Fc)
    for algo in "ghxy":
        for force in ("grid", "block"):
            r = engine.run(g, algo=algo, warp=32, force=force)
            assert np.array_equal(r.labels, lab[1:]) and r.num_sccs == n, (algo, force)
    b = scc.Batch(engine, [g])
    try:
        for cluster in (1, 4):
            b.set_cluster(cluster, 32)
            for algo in "gh":
                labels, res, _ = b.run(algo=algo)
                assert res[0][0] == n and np.array_equal(b.labels_of(labels, 0), lab[1:]), (algo, cluster)
    finally:
        b.close()
