"""Vertex states are packed eight to a word and walked 32 to a unit: sizes
around both, all drivers, both launch paths, against the sequential Tarjan
(labels are whole numbers: equal).  The graphs mix a giant SCC, trimmed
vertices, leftovers, a hub whose lists exceed what a lane tests alone, and
long paths that a warp follows by itself."""
import numpy as np
import pytest

import detectingscc_b200 as scc

pytestmark = pytest.mark.gpu


def _mixed(V, seed):
    rng = np.random.default_rng(seed)
    s, d = rng.integers(1, V + 1, 2 * V), rng.integers(1, V + 1, 2 * V)
    hub = int(rng.integers(1, V + 1))
    near = rng.integers(1, V + 1, min(V, 300))
    path = rng.permutation(V)[:V // 2] + 1            # a long path, closed on every other seed
    parts = [(s, d), (np.full(near.size, hub), near), (near[: near.size // 2], np.full(near.size // 2, hub)),
             (path[:-1], path[1:])]
    if seed % 2 and path.size > 1:
        parts.append((path[-1:], path[:1]))
    keep = rng.random(V + 1) < 0.8                    # a fifth of the vertices get no random arc
    a, b = (np.concatenate([p[i] for p in parts]) for i in (0, 1))
    ok = keep[a] & keep[b]
    return scc.graph_from_arcs(V, a[ok], b[ok])


@pytest.fixture(scope="module")
def engine():
    e = scc.Engine(0)
    yield e
    e.close()


@pytest.mark.parametrize("V", [1, 2, 7, 8, 9, 31, 32, 33, 63, 64, 65, 255, 256, 1023, 1025, 20000])
def test_unit_edges(engine, oracle_lib, V):
    for seed in (0, 1):
        g = _mixed(V, seed)
        lab, n = oracle_lib.tarjan(g.V, g.Fr, g.Fc)
        for algo, w, t1, t2 in (("g", 1, True, True), ("g", 1, False, True), ("h", 1, True, False), ("h", 1, False, False),
                                ("x", 8, True, False), ("y", 2, True, True)):
            for force in ("grid", "block"):
                r = engine.run(g, algo=algo, warp=w, t1=t1, t2=t2, force=force)
                assert np.array_equal(r.labels, lab[1:]) and r.num_sccs == n, (seed, algo, t1, t2, force)
