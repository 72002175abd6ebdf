"""Passes of the first search that stay one level (a fast growing search) and
passes in which warps go on with their own finds, on both sides of the rule.
Labels are whole numbers: they equal the sequential Tarjan's."""
import numpy as np
import pytest

import detectingscc_b200 as scc

pytestmark = pytest.mark.gpu


def _random(V, degree):
    rng = np.random.default_rng([V, degree])
    return scc.graph_from_arcs(V, rng.integers(1, V + 1, V * degree), rng.integers(1, V + 1, V * degree))


@pytest.fixture(scope="module")
def engine():
    e = scc.Engine(0)
    yield e
    e.close()


# one CTA: 256 arcs for each of 32 warps are reached from V = 1,366 on at degree 4
@pytest.mark.parametrize("V,degree", [(1365, 4), (1367, 4), (8000, 1), (8000, 2), (8000, 8), (16000, 16)])
def test_labels(engine, oracle_lib, V, degree):
    g = _random(V, degree)
    lab, n = oracle_lib.tarjan(g.V, g.Fr, g.Fc)
    for algo in "ghxy":
        for force in ("grid", "block"):
            r = engine.run(g, algo=algo, warp=4, force=force)
            assert np.array_equal(r.labels, lab[1:]) and r.num_sccs == n, (algo, force)
    b = scc.Batch(engine, [g, g])
    try:
        for cluster in (1, 4):
            b.set_cluster(cluster, 32)
            for algo in "gh":
                labels, res, _ = b.run(algo=algo)
                assert res[1][0] == n and np.array_equal(b.labels_of(labels, 1), lab[1:]), (algo, cluster)
    finally:
        b.close()


@pytest.mark.parametrize("seed", range(5))
def test_bottom_up_is_reached(engine, seed):
    """8,000 vertices of degree 9 on one CTA: with bottom-up steps half as
    many arcs are looked at as there are; a search that runs past them walks
    up to twice as many (forward and backward)."""
    rng = np.random.default_rng([8000, 9, seed])
    g = scc.graph_from_arcs(8000, rng.integers(1, 8001, 72000), rng.integers(1, 8001, 72000))
    r = engine.run(g, algo="h", force="block", instrument=True)
    assert r.stats["edges_scanned"] < g.E
