"""Colour peels: graphs whose SCCs the first search and the trims leave.

Chains of SCCs (each a cycle of 2 to 9 vertices, linked forward) with ids
that rise along the chain, fall along it, or are permuted; sizes around a
warp's item (32), above the residual solver's limit (4,096 vertices) and with
a hub above the chunk threshold (256 arcs) in one of the SCCs.  Labels are
whole numbers: they equal the sequential Tarjan's."""
import numpy as np
import pytest

import detectingscc_b200 as scc

pytestmark = pytest.mark.gpu


def _chain(V, order, hub, seed=5):
    rng = np.random.default_rng(seed)
    cuts = np.unique(np.concatenate([[0], np.cumsum(rng.integers(2, 10, V)), [V]]))
    cuts = cuts[cuts <= V]
    s, d = [], []
    for a, b in zip(cuts[:-1], cuts[1:]):
        p = np.arange(a, b)
        if b - a > 1:
            s.append(p)
            d.append(np.roll(p, -1))
        if b < V:   # to the next block and to one further on
            s.append([b - 1, a])
            d.append([b, min(V - 1, b + int(rng.integers(0, 40)))])
    if hub:         # one vertex with many arcs both ways inside one block of 700, placed in the middle
        m, n = V // 2, min(700, V // 3)
        p = np.arange(m, m + n)
        s += [np.full(n, m), p]
        d += [p, np.full(n, m)]
    s, d = np.concatenate(s).astype(np.int64), np.concatenate(d).astype(np.int64)
    ids = {"up": np.arange(V), "down": np.arange(V)[::-1], "mixed": rng.permutation(V)}[order] + 1
    return scc.graph_from_arcs(V, ids[s], ids[d])


@pytest.fixture(scope="module")
def engine():
    e = scc.Engine(0)
    yield e
    e.close()


@pytest.mark.parametrize("order", ["up", "down", "mixed"])
@pytest.mark.parametrize("V,hub", [(33, False), (1025, True), (4127, False), (9001, True), (33001, True)])
def test_chains_of_sccs(engine, oracle_lib, V, order, hub):
    g = _chain(V, order, hub)
    lab, n = oracle_lib.tarjan(g.V, g.Fr, g.Fc)
    for algo, w, t1 in (("g", 1, True), ("h", 1, True), ("x", 4, False), ("y", 8, False)):
        for force in ("grid", "block"):
            r = engine.run(g, algo=algo, warp=w, t1=t1, force=force)
            assert np.array_equal(r.labels, lab[1:]) and r.num_sccs == n, (algo, force)
    b = scc.Batch(engine, [g, g])
    try:
        for cluster in (1, 4):
            b.set_cluster(cluster, 32)
            labels, res, _ = b.run(algo="g")
            for i in range(2):
                assert res[i][0] == n and np.array_equal(b.labels_of(labels, i), lab[1:]), cluster
    finally:
        b.close()
