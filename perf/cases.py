"""The work that users of this framework have it do, as cases to be timed.

A case is a dict of plain values; ``prepare`` makes what a user's program holds
before the call (the resident graph, its seed MIS, the update batches), ``run``
is one pass through the public entry points, as such a program calls them.

Every case that updates a graph holds a short cycle of batches: ``cycle`` toggle
batches and then their inverses in reverse order, one batch a pass.  Links that
come and go keep the overlay at the size of a few batches however often the
case is run, while the membership and the cluster ids go on from pass to pass
as they do in a service.

Outputs are memberships, flags, line ids and counters: whole numbers, which the
library defines exactly.  There are no floating outputs, so no ``exact``.
"""
import math
import os
import random
import tempfile

import numpy as np
import torch

from misfit_gb300 import native
from misfit_gb300 import workloads as W

# the counters of a batch that describe the result, not how it was computed
COUNTERS = ("updates", "sub_batches", "seeds", "candidates", "clusters", "processed_edges", "max_csr")


def listed():
    return [
        # the smallest request of the serving stream: a handful of links of one small mesh
        {"name": "mesh1k_10", "kind": "plain", "graph": "rgg", "n": 1000, "degree": 8.0, "batch": 10,
         "endpoints": "low_degree", "exact_mode": False, "inputs": "host"},
        # the small plain configuration: ER(10,000, 8), files of 2,000 toggles
        {"name": "er10k_2000", "kind": "plain", "graph": "er", "n": 10000, "degree": 8.0, "batch": 2000,
         "endpoints": "uniform", "exact_mode": False, "inputs": "host"},
        # an ordinary request of the serving stream, odd sizes, endpoints of low degree
        {"name": "mesh100k_1003", "kind": "plain", "graph": "rgg", "n": 99991, "degree": 16.0, "batch": 1003,
         "endpoints": "low_degree", "exact_mode": False, "inputs": "host"},
        # the largest request of the batched and served streams
        {"name": "mesh1m_50000", "kind": "plain", "graph": "rgg", "n": 1000000, "degree": 20.0, "batch": 50000,
         "endpoints": "uniform", "exact_mode": False, "inputs": "host"},
        # a medium social-network-like graph with hubs, endpoints by degree
        {"name": "rmat17_pref_5003", "kind": "plain", "graph": "rmat", "n": 1 << 17, "degree": 16.0, "batch": 5003,
         "endpoints": "preferential", "exact_mode": False, "inputs": "host"},
        # exact-MIS mode with the batch already on the device
        {"name": "rmat20_exact_20000", "kind": "plain", "graph": "rmat", "n": 1 << 20, "degree": 16.0, "batch": 20000,
         "endpoints": "uniform", "exact_mode": True, "inputs": "device"},
        # the plain configuration at scale (the benchmark's own workload)
        {"name": "rmat22_100000", "kind": "plain", "graph": "rmat", "n": 1 << 22, "degree": 16.0, "batch": 100000,
         "endpoints": "uniform", "exact_mode": False, "inputs": "host"},
        # the pipelined loop: the next batch is launched before the last is collected
        {"name": "async_mesh300k_4x5000", "kind": "async", "graph": "rgg", "n": 300007, "degree": 12.0, "batch": 5000,
         "endpoints": "uniform", "depth": 4},
        # many graphs, one batch each, in one step
        {"name": "batched_48", "kind": "batched", "graphs": 48, "n_max": 1000000, "batch_max": 50000},
        # the serving pool: requests to many resident graphs at once
        {"name": "pool_24_64", "kind": "pool", "graphs": 24, "n_max": 300000, "requests": 64, "batch_max": 20000,
         "workers": 8},
        # a batch file parsed and flagged against the resident graph
        {"name": "parse_rmat20_200k", "kind": "parse", "graph": "rmat", "n": 1 << 20, "degree": 16.0, "batch": 200000},
        # the seed MIS of a graph, computed once per deployment
        {"name": "greedy_rmat21", "kind": "greedy", "graph": "rmat", "n": 1 << 21, "degree": 16.0},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["plain", "plain", "plain", "plain", "plain", "async", "batched", "pool", "parse", "greedy"])
    if kind == "batched":
        return {"kind": kind, "graphs": _log(rng, 6, 48), "n_max": _log(rng, 10000, 1000000),
                "batch_max": _log(rng, 500, 50000)}
    if kind == "pool":
        return {"kind": kind, "graphs": _log(rng, 4, 24), "n_max": _log(rng, 10000, 300000),
                "requests": _log(rng, 8, 64), "batch_max": _log(rng, 500, 20000), "workers": rng.choice([2, 4, 8])}
    graph = rng.choice(["rgg", "rgg", "er", "rmat"])
    if graph == "rmat":
        n, degree = 1 << rng.randint(13, 20), 16.0
    elif graph == "er":
        n, degree = _log(rng, 1000, 100000), round(rng.uniform(4, 16), 1)
    else:
        n, degree = _log(rng, 1000, 1000000), round(rng.uniform(4, 32), 1)
    if kind == "greedy":
        return {"kind": kind, "graph": graph, "n": n, "degree": degree}
    # a batch toggles at most a small share of the links
    most = max(20, min(50000, int(n * degree / 40)))
    batch = _log(rng, 10, most)
    if kind == "parse":
        return {"kind": kind, "graph": graph, "n": n, "degree": degree, "batch": _log(rng, 1000, 200000)}
    case = {"kind": kind, "graph": graph, "n": n, "degree": degree, "batch": batch,
            "endpoints": rng.choice(["uniform", "preferential", "low_degree"] if graph != "rmat" else
                                    ["uniform", "preferential"])}
    if kind == "async":
        return dict(case, batch=max(10, batch // 4), depth=rng.choice([2, 4]))
    return dict(case, exact_mode=rng.random() < 0.2, inputs=rng.choice(["host", "host", "device"]))


# ---- what a program has in hand before the call ----------------------------------

CYCLE = 2   # batches of a cycle before it turns back


def _graph(family, n, degree, seed):
    if family == "rmat":
        return W.rmat_graph_torch(n.bit_length() - 1, int(degree), seed)[1]
    if family == "er":
        return W.er_graph(n, degree, seed)
    return W.rgg_graph_torch(n, degree, seed)


def _cycle(nindex, nlist, seed, sizes, endpoints):
    """Toggle batches of the given sizes, then their inverses in reverse order: (u, v, ins) host arrays."""
    toggles = W.DeviceToggles(nindex, nlist, seed)
    there = [toggles.next_batch(m, endpoints=endpoints) for m in sizes]
    back = [(np.ascontiguousarray(u[::-1]), np.ascontiguousarray(v[::-1]), np.ascontiguousarray(1 - ins[::-1]))
            for u, v, ins in reversed(there)]
    return there + back


def _resident(nindex, nlist):
    g = native.Graph.from_csr(nindex, nlist)
    g.set_mis(g.greedy_mis())
    return g


class _Served:
    """A pool that is closed with the state that holds it."""

    def __init__(self, workers):
        self.pool = native.Pool(1 << 37, workers=workers)

    def __del__(self):
        self.pool.close()


class _File:
    """A batch file that is removed with the state that holds it."""

    def __init__(self, u, v):
        fd, self.path = tempfile.mkstemp(suffix=".mtx")
        os.close(fd)
        W.write_batch_file(self.path, u, v)

    def __del__(self):
        os.unlink(self.path)


def _many(case, seed):
    """The graphs of the batched and served streams: RGGs of log-uniform size, mean degree 4..32.  The sizes
    (of the batches too) are the case's, the points and the toggles the seed's."""
    rng = np.random.default_rng(case["graphs"])
    for k in range(case["graphs"]):
        n = int(round(math.exp(rng.uniform(math.log(1000), math.log(case["n_max"])))))
        yield k, rng, W.rgg_graph_torch(n, float(rng.uniform(4, 32)), seed * 1000 + k)


def _size(rng, most, entries):
    """Log-uniform batch size, at most half as many lines as the graph has links."""
    return min(int(round(math.exp(rng.uniform(math.log(10), math.log(most))))), max(10, entries // 4))


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case, "at": 0}
    if kind == "batched":
        s["graphs"], cycles = [], []
        for k, rng, (nindex, nlist) in _many(case, seed):
            s["graphs"].append(_resident(nindex, nlist))
            sizes = [_size(rng, case["batch_max"], nlist.size)] * CYCLE
            cycles.append(_cycle(nindex, nlist, seed + k, sizes, "low_degree" if k % 2 == 0 else "uniform"))
        s["steps"] = [list(step) for step in zip(*cycles)]
        return s
    if kind == "pool":
        s["served"] = _Served(case["workers"])
        pool, cycles = s["served"].pool, {}
        ranks = None
        for k, rng, (nindex, nlist) in _many(case, seed):
            with native.Graph.from_csr(nindex, nlist) as g:
                mis = g.greedy_mis()
            gid = pool.add_graph(nindex, nlist, mis)
            ranks = rng
            sizes = [_size(rng, case["batch_max"], nlist.size) for _ in range(CYCLE)]
            cycles[gid] = _cycle(nindex, nlist, seed + k, sizes, ("uniform", "preferential", "low_degree")[k % 3])
        # requests choose their graph by Zipf(1.1); each graph walks its own cycle
        gids = sorted(cycles)
        p = np.arange(1, len(gids) + 1) ** -1.1
        s["requests"] = [gids[j] for j in ranks.choice(len(gids), size=case["requests"], p=p / p.sum())]
        s["cycles"], s["next"], s["gids"] = cycles, {g: 0 for g in gids}, gids
        return s
    nindex, nlist = _graph(case["graph"], case["n"], case["degree"], seed)
    if kind == "greedy":
        s["graph"] = native.Graph.from_csr(nindex, nlist)
        return s
    if kind == "parse":
        u, v, _ = W.DeviceToggles(nindex, nlist, seed + 1).next_batch(case["batch"])
        s["graph"], s["file"] = native.Graph.from_csr(nindex, nlist), _File(u, v)
        return s
    s["graph"] = _resident(nindex, nlist)
    sizes = [case["batch"]] * CYCLE
    s["batches"] = _cycle(nindex, nlist, seed + 1, sizes, case["endpoints"])
    if kind == "plain":
        s["graph"].set_exact(case["exact_mode"])
        if case["inputs"] == "device":
            s["batches"] = [tuple(torch.as_tensor(a, device="cuda") for a in b) for b in s["batches"]]
    return s


# ---- one pass -----------------------------------------------------------------


def run(s):
    case, kind = s["case"], s["case"]["kind"]
    if kind == "plain":
        g = s["graph"]
        u, v, ins = s["batches"][s["at"] % len(s["batches"])]
        s["at"] += 1
        if case["inputs"] == "device":
            g.apply_batch_device(u.data_ptr(), v.data_ptr(), ins.data_ptr(), u.numel())
        else:
            g.apply_batch(u, v, ins)
        st = g.stats()
        return {"mis": g.get_mis(), "counters": np.array([st[k] for k in COUNTERS], np.int64)}
    if kind == "async":
        g, got = s["graph"], []
        for k in range(case["depth"]):
            g.apply_batch_async(*s["batches"][s["at"] % len(s["batches"])])
            s["at"] += 1
            if k:
                got.append(g.collect())
        got.append(g.collect())
        return {"mis": g.get_mis(), "counters": np.array([[st[k] for k in COUNTERS] for st in got], np.int64)}
    if kind == "batched":
        native.apply_batches(s["graphs"], s["steps"][s["at"] % len(s["steps"])])
        s["at"] += 1
        return {"mis": np.concatenate([g.get_mis() for g in s["graphs"]])}
    if kind == "pool":
        pool = s["served"].pool
        ids = []
        for gid in s["requests"]:
            cycle = s["cycles"][gid]
            u, v, ins = cycle[s["next"][gid] % len(cycle)]
            s["next"][gid] += 1
            ids.append(pool.submit(gid, u, v, ins))
        for rid in ids:
            pool.wait(rid)
        return {"mis": np.concatenate([pool.get_mis(gid) for gid in s["gids"]])}
    if kind == "parse":
        u, v, ins = s["graph"].parse_batch_file(s["file"].path)
        return {"u": u, "v": v, "ins": ins}
    return {"mis": s["graph"].greedy_mis()}


# ---- what a pass cannot do without ----------------------------------------------


def _update_bytes(n, degree, m):
    """The batch (two ids and a flag a line), the membership out, the rows of the touched endpoints and of their
    neighbours once, and the id and membership of every vertex of those rows once."""
    reached = min(n, 2 * m * (1 + degree))
    around = min(n, 2 * m * (1 + degree) ** 2)
    return 9.0 * m + n + (4.0 * degree + 8.0) * reached + 5.0 * around


def work(case):
    kind = case["kind"]
    if kind in ("batched", "pool"):
        rng = random.Random(1)   # means over the drawn graphs and sizes
        total, count = 0.0, case["graphs"] if kind == "batched" else case["requests"]
        for _ in range(count):
            total += _update_bytes(_log(rng, 1000, case["n_max"]), rng.uniform(4, 32), _log(rng, 10, case["batch_max"]))
        return {"bytes": total, "flops": 0}
    n = case["n"]
    degree = case["degree"] * (2 if case["graph"] == "rmat" else 1)   # R-MAT: samples per vertex, both directions
    if kind == "plain":
        return {"bytes": _update_bytes(n, degree, case["batch"]), "flops": 0}
    if kind == "async":
        return {"bytes": case["depth"] * _update_bytes(n, degree, case["batch"]), "flops": 0}
    if kind == "parse":   # the text in (about 14 bytes a line), ids and flags out, one probe of a row for a line
        return {"bytes": case["batch"] * (14.0 + 9.0 + 32.0), "flops": 0}
    return {"bytes": n * (4.0 * degree + 8.0) + n, "flops": 0}   # greedy: every row once
