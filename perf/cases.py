"""The work that users of this engine have it do, as cases that can be timed.

Every pass goes through the public Python API (``Engine``, ``Batch``,
``Server``).  A case names a path (``what``), a graph family with its sizes,
and the driver's options:

* ``device``  one decomposition of a CSR that is already on the GPU, labels
              left there (``Engine.run_device``)
* ``host``    the forward CSR in page-locked host memory, labels back there
              (``Engine.run`` with the reverse CSR built on the device)
* ``file``    a GTgraph text file to labels (``Engine.load_graph_device``,
              then ``Engine.run_device``)
* ``derive``  the reverse CSR of a device-resident forward CSR
* ``batch``   many independent graphs resident on the GPU, one launch
* ``serve``   a burst of requests through the request server

Graphs come from ``detectingscc_b200.graphs`` and a seed.
"""
import functools
import math
import tempfile

import numpy as np
import torch

import detectingscc_b200 as scc
from detectingscc_b200 import graphs

DEV = "cuda"


def listed():
    return [
        # The smallest call: the reference's own use, one GTgraph random graph
        # of about a thousand vertices through vHong.  Latency counts.
        {"name": "planted_1k_vhong", "what": "device", "family": "random", "V": 1024, "m": 4096, "cycles": 16,
         "algo": "g", "t1": True, "t2": False, "w": 1},
        # An ordinary sparse random graph of ragged size, just above what one
        # CTA takes: short whole-GPU passes.
        {"name": "random_50k_vslota", "what": "device", "family": "random", "V": 50021, "m": 200083, "cycles": 16,
         "algo": "h", "t1": True, "t2": True, "w": 1},
        # A road-like graph of a city's size: high diameter, many light levels.
        {"name": "grid_701_vhong", "what": "device", "family": "grid", "n": 701, "algo": "g", "t1": True, "t2": True,
         "w": 1},
        # A web- or social-like graph whose ids do not follow degree, through
        # Hong's driver with both trims, virtual warps of eight.
        {"name": "rmat_s20p_whong8", "what": "device", "family": "rmat", "scale": 20, "factor": 16, "permute": True,
         "algo": "x", "t1": True, "t2": True, "w": 8},
        # The headline workload: R-MAT scale 22 through vSlota.
        {"name": "rmat_s22_vslota", "what": "device", "family": "rmat", "scale": 22, "factor": 16, "permute": False,
         "algo": "h", "t1": True, "t2": True, "w": 1},
        # The largest road-like graph: 16.8M vertices, wSlota with -w 8.
        {"name": "grid_4096_wslota8", "what": "device", "family": "grid", "n": 4096, "algo": "y", "t1": True,
         "t2": True, "w": 8},
        # End to end from host memory: a million-vertex graph crosses PCIe.
        {"name": "host_rmat_s20_vslota", "what": "host", "family": "rmat", "scale": 20, "factor": 16,
         "permute": False, "algo": "h", "t1": True, "t2": True, "w": 1},
        # The command line's work: a GTgraph text file to labels.
        {"name": "file_rmat_s16_vhong", "what": "file", "family": "rmat", "scale": 16, "factor": 16,
         "permute": False, "algo": "g", "t1": True, "t2": False, "w": 1},
        # A program that holds only the forward CSR builds the reverse one.
        {"name": "derive_rmat_s21", "what": "derive", "family": "rmat", "scale": 21, "factor": 16, "permute": False},
        # Many small graphs at once, as a per-function or per-module analysis
        # has them; default schedule.
        {"name": "batch_2048_small_vslota", "what": "batch", "n": 2048, "vmin": 64, "vmax": 4096, "algo": "h",
         "t1": True, "t2": True, "w": 1, "tune": False},
        # Graphs of very uneven sizes, kept resident and run many times: the
        # batch is autotuned once.
        {"name": "batch_512_mixed_vhong", "what": "batch", "n": 512, "vmin": 64, "vmax": 65536, "algo": "g",
         "t1": True, "t2": True, "w": 1, "tune": True},
        # A burst of requests of the mix, two larger graphs among them.
        {"name": "serve_burst_vhong", "what": "serve", "n": 96, "vmin": 64, "vmax": 65536, "big": 2, "scale": 17,
         "algo": "g", "t1": True, "t2": True, "w": 1},
    ]


def draw(rng):
    def logint(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    algo = rng.choice("ghxy")
    opts = {"algo": algo, "t1": True, "t2": rng.random() < 0.7, "w": rng.choice([1, 2, 4, 8, 16, 32])}
    if algo in "hy" and rng.random() < 0.2:
        opts["t1"] = False
    what = rng.choice(["device"] * 8 + ["host", "file", "derive", "batch", "batch", "serve"])
    if what == "batch":
        vmax = rng.choice([2048, 8192, 65536])
        return {"what": what, "n": logint(24, {2048: 3000, 8192: 1200, 65536: 400}[vmax]), "vmin": 64, "vmax": vmax,
                "tune": rng.random() < 0.5, **opts}
    if what == "serve":
        return {"what": what, "n": logint(8, 90), "vmin": 64, "vmax": rng.choice([4096, 65536]),
                "big": rng.randint(0, 2), "scale": rng.randint(15, 17), **opts}
    small = {"device": 1.0, "host": 0.25, "derive": 0.5, "file": 0.02}[what]
    family = rng.choice(["random", "rmat", "rmat"] + ["grid"] * (what != "derive"))
    if family == "random":
        V = logint(200, 2000000 * small)
        g = {"V": V, "m": int(V * rng.uniform(1.2, 12.0)), "cycles": rng.randint(0, 24) if what != "derive" else 0}
    elif family == "rmat":
        g = {"scale": rng.randint(9, 21 + int(round(math.log2(small)))), "factor": rng.randint(4, 16),
             "permute": rng.random() < 0.5}
    else:
        g = {"n": logint(20, 2600 * math.sqrt(small))}
    return {"what": what, "family": family, **g, **({} if what == "derive" else opts)}


def _arcs(case, seed):
    """(V, src, dst) of the case's graph, 1-based int64 arcs on the GPU."""
    if case["family"] == "random":
        return graphs.planted_random(case["V"], case["m"], case["cycles"], 4, min(32, case["V"]), seed=seed, device=DEV)
    if case["family"] == "rmat":
        # the reverse CSR keeps duplicates and self-loops, as a GTgraph file may hold them
        return graphs.rmat(case["scale"], case["factor"], seed=seed, device=DEV, permute=case["permute"],
                           clean=case["what"] != "derive")
    return graphs.grid(case["n"], seed=seed, device=DEV)


def _mix(case, seed):
    """The arcs of every graph of a batch or of a burst, in order: vertex
    counts spread evenly over the logarithm of their range, degrees and arcs
    drawn from the seed."""
    n, lo, hi = case["n"], case["vmin"], case["vmax"]
    sizes = [int(round(lo * (hi / lo) ** (((i * 0.6180339887) % 1.0)))) for i in range(n)]
    out = [graphs.batch_mix_graph(i, V, V, seed=seed) for i, V in enumerate(sizes)]
    for i in range(case.get("big", 0)):
        V, s, d = graphs.rmat(case["scale"], 16, seed=seed + 1 + i, device=DEV)
        out.append((V, s.cpu().numpy(), d.cpu().numpy()))
    return out


def _pinned(a):
    """The same values in page-locked host memory."""
    return torch.from_numpy(np.ascontiguousarray(a).view(np.int32)).pin_memory().numpy().view(np.uint32)


@functools.lru_cache(maxsize=None)
def _engine():
    return scc.Engine(0)


@functools.lru_cache(maxsize=None)
def _server(algo, t1, t2, w):
    return scc.Server(0, algo=algo, t1=t1, t2=t2, warp=w)


def _opts(case):
    return {"algo": case["algo"], "t1": case["t1"], "t2": case["t2"], "warp": case["w"]}


def prepare(case, seed):
    what = case["what"]
    s = {"what": what, "eng": _engine()}
    if what in ("batch", "serve"):
        gs = [scc.graph_from_arcs(*g) for g in _mix(case, seed)]
        if what == "batch":
            s["batch"] = scc.Batch(s["eng"], gs)
            s["out"] = _pinned(np.zeros(s["batch"].total_vertices, np.uint32))
            if case["tune"]:
                s["batch"].autotune(**_opts(case))
        else:
            s["graphs"] = [scc.Graph(g.V, g.E, *map(_pinned, (g.Fr, g.Fc, g.Br, g.Bc))) for g in gs]
            s["out"] = [np.zeros(g.V, np.uint32) for g in gs]
            s["server"] = _server(case["algo"], case["t1"], case["t2"], case["w"])
        s["opts"] = _opts(case)
        return s
    V, src, dst = _arcs(case, seed)
    s["V"], s["E"] = V, int(src.shape[0])
    if what == "file":
        g = graphs.to_graph(V, src, dst)
        s["file"] = tempfile.NamedTemporaryFile(suffix=".gr")   # removed with the state
        scc.save_gtgraph(s["file"].name, g)
    else:
        Fr, Fc, Br, Bc = graphs.csr_from_arcs_torch(V, src, dst)
        if what == "host":
            none = np.zeros(0, np.uint32)
            s["graph"] = scc.Graph(V, s["E"], _pinned(Fr.cpu().numpy()), _pinned(Fc.cpu().numpy()), none, none)
        elif what == "derive":
            s["csr"] = (Fr, Fc, torch.empty_like(Br), torch.empty_like(Bc))
        else:
            s["csr"] = (Fr, Fc, Br, Bc)
    if what != "derive":
        s["opts"] = _opts(case)
        s["out"] = (_pinned(np.zeros(V, np.uint32)) if what == "host" else
                    torch.empty(V, dtype=torch.int32, device=DEV))
    return s


def _counts(r):
    return [r.num_sccs, r.num_trim1, r.num_trim2, r.num_pivot]


def run(s):
    what, eng = s["what"], s["eng"]
    if what == "device":
        r = eng.run_device(s["V"], s["E"], *s["csr"], labels_out=s["out"], **s["opts"])
        return {"labels": s["out"], "counts": _counts(r)}
    if what == "host":
        r = eng.run(s["graph"], out=s["out"], derive_reverse=True, **s["opts"])
        return {"labels": s["out"], "counts": _counts(r)}
    if what == "file":
        V, E, Fr, Fc, Br, Bc = eng.load_graph_device(s["file"].name)
        r = eng.run_device(V, E, Fr, Fc, Br, Bc, labels_out=s["out"], **s["opts"])
        return {"labels": s["out"], "counts": _counts(r)}
    if what == "derive":
        eng.derive_reverse(s["V"], s["E"], *s["csr"])
        return {"Br": s["csr"][2], "Bc": s["csr"][3]}
    if what == "batch":
        labels, results, _ = s["batch"].run(out=s["out"], **s["opts"])
        return {"labels": labels, "results": np.array(results, np.int64)}
    tickets = {s["server"].submit(g, o): i for i, (g, o) in enumerate(zip(s["graphs"], s["out"]))}
    results = np.zeros((len(tickets), 3), np.int64)
    left = len(tickets)
    while left:
        for r in s["server"].poll(wait_ms=1000):
            results[tickets[r["ticket"]]] = r["num_sccs"], r["num_trim1"], r["status"]
            left -= 1
    return {"labels": np.concatenate(s["out"]), "results": results}


def _size(case):
    """Vertices and arcs of the case's graph or graphs (their mean over seeds)."""
    if case["what"] in ("batch", "serve"):
        # half the graphs have about 10 arcs a vertex, half about 6.9; V is log-uniform
        V = case["n"] * (case["vmax"] - case["vmin"]) / math.log(case["vmax"] / case["vmin"])
        big = case.get("big", 0) * 2.0 ** case.get("scale", 0)
        return V + big, 8.4 * V + 15.0 * big
    if case["family"] == "random":
        return case["V"], case["m"] + 18 * case["cycles"]
    if case["family"] == "rmat":
        return 2.0 ** case["scale"], 0.95 * case["factor"] * 2.0 ** case["scale"]
    return case["n"] ** 2, 2 * case["n"] * (case["n"] - 1) * 1.7


def work(case):
    V, E = _size(case)
    what = case["what"]
    if what == "derive":
        b = 2 * 4 * (V + E)
    elif what == "host":      # the forward CSR in, the labels out
        b = 4 * (V + E) + 4 * V
    elif what == "file":      # "a u v 1" a line
        b = E * (6 + 2 * (math.log10(V) + 0.5)) + 4 * V
    else:                     # both CSRs in, the labels out
        b = 2 * 4 * (V + E) + 4 * V
    return {"bytes": float(b), "flops": 0.0}


def _exact_labels(V, src, dst):
    """Smallest vertex id of every vertex's SCC (entry v - 1), by forward and
    backward maxima: two vertices of one SCC are reached by the same largest id
    and reach the same largest id; arcs between vertices that differ in either
    are dropped until none is left."""
    ids = torch.arange(V + 1, dtype=torch.int64, device=src.device)

    def spread(a, b):
        m = ids.clone()
        while True:
            n = m.scatter_reduce(0, b, m[a], "amax")
            n = torch.maximum(n, n[n])
            if torch.equal(n, m):
                return m
            m = n

    while True:
        f, b = spread(src, dst), spread(dst, src)
        keep = (f[src] == f[dst]) & (b[src] == b[dst])
        if bool(keep.all()):
            break
        src, dst = src[keep], dst[keep]
    low = torch.full_like(ids, V + 1).scatter_reduce(0, f, ids, "amin")
    return low[f][1:]


def exact(case, seed):
    what = case["what"]
    if what in ("batch", "serve"):
        base, srcs, dsts, sizes = 0, [], [], []
        for V, s, d in _mix(case, seed):
            srcs.append(s + base)
            dsts.append(d + base)
            sizes.append(V)
            base += V
        src, dst = (torch.from_numpy(np.concatenate(x).astype(np.int64)).to(DEV) for x in (srcs, dsts))
        starts = torch.tensor(np.repeat(np.concatenate([[0], np.cumsum(sizes)[:-1]]), sizes), device=DEV)
        labels = _exact_labels(base, src, dst) - starts
        return {"labels": labels, "results": None}
    V, src, dst = _arcs(case, seed)
    if what == "derive":
        d, s = (lambda k: (k // (V + 1), k % (V + 1)))(torch.sort(dst * (V + 1) + src).values)
        Br = torch.zeros(V + 2, dtype=torch.int64, device=DEV)
        Br[1:] = torch.cumsum(torch.bincount(d, minlength=V + 2), 0)[:V + 1]
        return {"Br": Br, "Bc": s}
    labels = _exact_labels(V, src, dst)
    num = int((labels == torch.arange(1, V + 1, device=DEV)).sum())
    return {"labels": labels, "counts": [num, None, None, None]}
