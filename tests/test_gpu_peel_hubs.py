"""Colour peels around vertices whose lists are cut into chunks.

A hub h points at many leaves, every leaf at z, and a path z, c[k], ..., c[0]
closes the cycle; ids h < c[0] < c[1] < ..., so one item of a warp raises h
again in every round that the warp goes on for by itself, and h's list may be
cut only once a pass.  A two-way star elsewhere takes the first pivot, and
two-cycles keep the remainder above the single-CTA tail.  Labels are whole
numbers: they equal the sequential Tarjan's."""
import numpy as np
import pytest

import detectingscc_b200 as scc

pytestmark = pytest.mark.gpu


def _hub(nleaf, rev, chain=11, star=1000, pairs=1100):
    c = np.arange(2, 2 + chain)
    z = 2 + chain
    leaf = np.arange(z + 1, z + 1 + nleaf)
    s0 = z + 1 + nleaf
    st = np.arange(s0 + 1, s0 + 1 + star)
    p = np.arange(s0 + 1 + star, s0 + 1 + star + 2 * pairs).reshape(-1, 2)
    src = [np.full(nleaf, 1), leaf, [z], c[1:], [c[0]], np.full(star, s0), st, p[:, 0], p[:, 1]]
    dst = [leaf, np.full(nleaf, z), [c[-1]], c[:-1], [1], st, np.full(star, s0), p[:, 1], p[:, 0]]
    src, dst = np.concatenate(src).astype(np.int64), np.concatenate(dst).astype(np.int64)
    return scc.graph_from_arcs(int(p.max()), *((dst, src) if rev else (src, dst)))


@pytest.fixture(scope="module")
def engine():
    e = scc.Engine(0)
    yield e
    e.close()


@pytest.mark.parametrize("rev", [False, True])
@pytest.mark.parametrize("nleaf", [257, 20000, 131072])
def test_hub_raised_every_round(engine, oracle_lib, nleaf, rev):
    g = _hub(nleaf, rev)
    lab, n = oracle_lib.tarjan(g.V, g.Fr, g.Fc)
    engine.set_tuning("tail_vertices", 0)
    engine.set_tuning("trace", 4096)
    try:
        for algo in "ghxy":
            for force in ("grid", "block"):
                r = engine.run(g, algo=algo, warp=8, force=force)
                assert np.array_equal(r.labels, lab[1:]) and r.num_sccs == n, (algo, force)
                if nleaf > 16384:   # more arcs than the residual solver takes
                    ran = {p for p, _, _ in engine.trace()}
                    assert {"prop", "peel_scc"} <= ran
    finally:
        engine.set_tuning("trace", 0)
        engine.set_tuning("tail_vertices", 1024)
    b = scc.Batch(engine, [g])
    try:
        for cluster in (1, 4, 16):
            b.set_cluster(cluster, 32)
            for algo in "gh":
                labels, res, _ = b.run(algo=algo)
                assert res[0][0] == n and np.array_equal(b.labels_of(labels, 0), lab[1:]), (algo, cluster)
    finally:
        b.close()
