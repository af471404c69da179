"""The work this library is measured on: what a user has it do, through its
public entry points (albba_gb300.Graph, Worklist, SellMatrix).

Five kinds of work (case["op"]):

  bfs       one breadth-first search from one root on a graph that is already
            resident and built: levels and parents into device arrays
  ms        the batched search from up to 64 roots, n x 64 levels on the device
  worklist  many small uneven graphs, several roots each, in one launch
  spmv      y = A x in fp64 with device vectors
  host      the whole way: CSR in page-locked host memory -> graph -> SELL
            build -> search -> levels (and parents) in host memory

Graphs are seeded and made on the GPU: R-MAT (.57/.19/.19/.05, ids permuted),
Erdos-Renyi, and a grid with a tenth of its edges dropped and a few
shortcuts. Undirected ones are symmetrised; duplicates and self-loops are
removed. Sizes follow the repository's own workloads (R-MAT scale 10 to 24 at
edge factors 4 to 32, the 4096 x 4096 grid, mean degree 8 for Erdos-Renyi)
and the ragged ones between them.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import albba_gb300 as ab
from albba_gb300 import selector


def listed():
    return [
        # the smallest call: a graph that fits in a corner of L2, where the
        # search is all latency and launches
        {"name": "bfs_rmat_1k", "op": "bfs", "graph": "rmat", "n": 1 << 10, "ef": 16,
         "policy": "beamer", "loop": "graph"},
        # the correctness workload's size (R-MAT scale 16), default options
        {"name": "bfs_rmat_64k", "op": "bfs", "graph": "rmat", "n": 1 << 16, "ef": 16,
         "policy": "beamer", "loop": "graph"},
        # an ordinary graph with a vertex count that no tile divides
        {"name": "bfs_rmat_1m_odd", "op": "bfs", "graph": "rmat", "n": 1_000_003, "ef": 8,
         "policy": "beamer", "loop": "graph"},
        # the headline graph searched one root at a time, shipped selector
        {"name": "bfs_rmat_16m", "op": "bfs", "graph": "rmat", "n": 1 << 24, "ef": 16,
         "policy": "learned", "loop": "graph"},
        # no hubs and more levels: uniform random graph, default options
        {"name": "bfs_er_4m", "op": "bfs", "graph": "er", "n": 1 << 22, "ef": 4,
         "policy": "beamer", "loop": "graph"},
        # hundreds of levels with small frontiers: the road-like case, on the
        # loop that is meant for it
        {"name": "bfs_grid_16m", "op": "bfs", "graph": "grid", "n": 1 << 24, "ef": 2,
         "policy": "learned", "loop": "persistent"},
        # a batch that is not full, on a graph whose state stays in L2
        {"name": "ms_rmat_64k_37", "op": "ms", "graph": "rmat", "n": 1 << 16, "ef": 16,
         "roots": 37, "policy": "beamer"},
        # the headline: 64 roots at once on R-MAT scale 24, shipped selector
        {"name": "ms_rmat_16m_64", "op": "ms", "graph": "rmat", "n": 1 << 24, "ef": 16,
         "roots": 64, "policy": "learned"},
        # uneven small graphs (scales 10 to 16, edge factors 4 to 32), 8 roots each
        {"name": "worklist_48x8", "op": "worklist", "graphs": 48, "roots": 8, "lo": 10, "hi": 16},
        # a small sparse system without hubs: one SpMV of an iterative method
        {"name": "spmv_er_20k", "op": "spmv", "graph": "er", "n": 20_011, "ef": 8,
         "values": "signed"},
        # power-law matrix with hub rows, large enough to leave L2
        {"name": "spmv_rmat_4m", "op": "spmv", "graph": "rmat", "n": 1 << 22, "ef": 16,
         "values": "signed"},
        # end to end from host memory, as the benchmark's second number
        {"name": "host_ms_rmat_1m", "op": "host", "graph": "rmat", "n": 1 << 20, "ef": 16,
         "form": "ms", "directed": False},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_graph(rng, lo, hi, kinds):
    kind = rng.choice(kinds)
    n = _log_int(rng, lo, hi)
    if kind == "grid":
        side = max(8, int(math.sqrt(n)))
        return {"graph": "grid", "n": side * side, "ef": 2}
    return {"graph": kind, "n": n, "ef": rng.choice([4, 8, 16]) if kind == "rmat" else 4}


def draw(rng):
    op = rng.choice(["bfs", "bfs", "bfs", "ms", "worklist", "spmv", "host"])
    if op == "bfs":
        c = _draw_graph(rng, 1 << 10, 1 << 24, ["rmat", "rmat", "er", "grid"])
        # long searches on the persistent loop, as the documentation has it;
        # the others on the default loop, or now and then on that one
        loop = "persistent" if c["graph"] == "grid" else rng.choice(["graph", "graph", "persistent"])
        return {"op": "bfs", **c, "policy": rng.choice(["beamer", "learned"]), "loop": loop}
    if op == "ms":
        c = _draw_graph(rng, 1 << 11, 12_000_000, ["rmat", "rmat", "er"])
        return {"op": "ms", **c, "roots": rng.choice([1, 17, 64, 64, rng.randint(2, 63)]),
                "policy": rng.choice(["beamer", "learned"])}
    if op == "worklist":
        lo = rng.randint(8, 12)
        return {"op": "worklist", "graphs": _log_int(rng, 8, 48), "roots": rng.randint(1, 8),
                "lo": lo, "hi": min(16, lo + rng.randint(1, 5))}
    if op == "spmv":
        c = _draw_graph(rng, 1 << 11, 4_000_000, ["rmat", "rmat", "er", "grid"])
        return {"op": "spmv", **c, "values": rng.choice(["signed", "positive"])}
    c = _draw_graph(rng, 1 << 12, 1 << 20, ["rmat", "er"])
    return {"op": "host", **c, "form": rng.choice(["ms", "bfs"]), "directed": rng.random() < 0.5}


# ------------------------------------------------------------------ inputs
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _rmat_edges(n, m, g):
    """m R-MAT edges over n vertices (bits of the next power of two, scaled
    down to n), 32 M at a time."""
    scale = max(1, (n - 1).bit_length())
    us, vs = [], []
    for i in range(0, m, 1 << 25):
        k = min(1 << 25, m - i)
        u = torch.zeros(k, dtype=torch.int64, device="cuda")
        v = torch.zeros(k, dtype=torch.int64, device="cuda")
        for _ in range(scale):
            r = torch.rand(k, device="cuda", generator=g)
            # quadrants a = .57, b = .19, c = .19, d = .05
            u.mul_(2).add_(r >= 0.76)
            v.mul_(2).add_(((r >= 0.57) & (r < 0.76)) | (r >= 0.95))
        if n != 1 << scale:
            u = (u * n) >> scale
            v = (v * n) >> scale
        us.append(u)
        vs.append(v)
    perm = torch.randperm(n, device="cuda", generator=g)
    return perm[torch.cat(us)], perm[torch.cat(vs)]


def _edges(kind, n, ef, g):
    if kind == "grid":
        side = int(round(math.sqrt(n)))
        at = torch.arange(n, device="cuda").view(side, side)
        u = torch.cat([at[:, :-1].reshape(-1), at[:-1].reshape(-1)])
        v = torch.cat([at[:, 1:].reshape(-1), at[1:].reshape(-1)])
        keep = torch.rand(u.shape[0], device="cuda", generator=g) >= 0.1
        cuts = max(1, n // 10_000)
        su, sv = torch.randint(0, n, (2, cuts), device="cuda", generator=g)
        return torch.cat([u[keep], su]), torch.cat([v[keep], sv])
    m = n * ef
    if kind == "er":
        u, v = torch.randint(0, n, (2, m), device="cuda", generator=g)
        return u, v
    return _rmat_edges(n, m, g)


def _csr(kind, n, ef, seed, directed=False):
    """(rowptr int64, col int32) on the GPU, rows ascending."""
    g = _gen(seed)
    u, v = _edges(kind, n, ef, g)
    keep = u != v
    u, v = u[keep], v[keep]
    key = u * n + v if directed else torch.cat([u * n + v, v * n + u])
    del u, v, keep
    key = torch.unique_consecutive(torch.sort(key).values)
    col = (key % n).to(torch.int32)
    deg = torch.bincount(key // n, minlength=n)
    del key
    rp = torch.zeros(n + 1, dtype=torch.int64, device="cuda")
    torch.cumsum(deg, 0, out=rp[1:])
    return rp, col, g


def _roots(rp, col, count, g):
    """Roots that are ends of stored edges (so that they have neighbours)."""
    at = torch.randint(0, col.shape[0], (count,), device="cuda", generator=g)
    return col[at].cpu().numpy().astype(np.int32)


def _host(rp, col):
    return ab.Csr(rp.cpu().numpy(), col.cpu().numpy())


def _pinned(t):
    h = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    h.copy_(t)
    return h.numpy()


def _resident(case, seed):
    rp, col, g = _csr(case["graph"], case["n"], case["ef"], seed)
    roots = _roots(rp, col, case.get("roots", 1), g)
    csr = _host(rp, col)
    del rp, col
    torch.cuda.empty_cache()
    dg = ab.Graph(csr, ab.CSR_SYMMETRIC | ab.CSR_SORTED)
    dg.sell_build()
    if case["policy"] == "learned":
        selector.install()
    return dg, roots


def _matrix(case, seed):
    """CSR with values and x on the GPU: signed as in the benchmark, or
    positive as in a random walk (each row's weights near 1 / its length)."""
    rp, col, g = _csr(case["graph"], case["n"], case["ef"], seed)
    n, nnz = case["n"], col.shape[0]
    if case["values"] == "signed":
        val = torch.rand(nnz, dtype=torch.float64, device="cuda", generator=g) * 2 - 1
        x = torch.randn(n, dtype=torch.float64, device="cuda", generator=g)
    else:
        deg = (rp[1:] - rp[:-1]).clamp(min=1).to(torch.float64)
        val = 1.0 / deg[col.long()]
        x = torch.rand(n, dtype=torch.float64, device="cuda", generator=g) / n
    return rp, col, val, x


def prepare(case, seed):
    op = case["op"]
    if op == "bfs":
        dg, roots = _resident(case, seed)
        return {"op": op, "g": dg, "root": int(roots[0]),
                "opts": ab.bfs_opts(case["policy"], case["loop"]),
                "level": torch.empty(case["n"], dtype=torch.int32, device="cuda"),
                "parent": torch.empty(case["n"], dtype=torch.int32, device="cuda")}
    if op == "ms":
        dg, roots = _resident(case, seed)
        return {"op": op, "g": dg, "roots": roots, "opts": ab.bfs_opts(case["policy"]),
                "levels": torch.empty((case["n"], 64), dtype=torch.int32, device="cuda")}
    if op == "worklist":
        rng = np.random.default_rng(seed)
        wl = ab.Worklist()
        for i in range(case["graphs"]):
            # scales spread evenly over the range, edge factors at random
            scale = case["lo"] + i % (case["hi"] - case["lo"] + 1)
            rp, col, g = _csr("rmat", 1 << scale, int(rng.choice([4, 8, 16, 32])),
                              int(rng.integers(1 << 40)))
            roots = _roots(rp, col, case["roots"], g)
            dg = ab.Graph(_host(rp, col), ab.CSR_SYMMETRIC | ab.CSR_SORTED)
            dg.sell_build()
            wl.add(dg, roots)
        return {"op": op, "wl": wl,
                "levels": torch.empty(wl.size()[0], dtype=torch.int32, device="cuda")}
    if op == "spmv":
        rp, col, val, x = _matrix(case, seed)
        m = ab.SellMatrix(rp.cpu().numpy(), col.cpu().numpy(), val.cpu().numpy())
        return {"op": op, "m": m, "x": x, "y": torch.empty_like(x)}
    rp, col, g = _csr(case["graph"], case["n"], case["ef"], seed, case["directed"])
    state = {"op": op, "form": case["form"], "roots": _roots(rp, col, 64, g),
             "csr": ab.Csr(_pinned(rp), _pinned(col)),
             "flags": ab.CSR_OUT if case["directed"] else ab.CSR_SYMMETRIC | ab.CSR_SORTED}
    if case["form"] == "ms":
        state["out"] = torch.empty((case["n"], 64), dtype=torch.int32, pin_memory=True).numpy()
    return state


# -------------------------------------------------------------------- runs
def run(s):
    op = s["op"]
    if op == "bfs":
        st = s["g"].bfs_device(s["root"], s["level"], s["parent"], s["opts"])
        return {"level": s["level"], "parent": s["parent"], "levels": st.num_levels,
                "reached": st.reached, "edges": st.edges}
    if op == "ms":
        st = s["g"].msbfs64_device(s["roots"], s["levels"], s["opts"])
        return {"levels": s["levels"], "depth": st.num_levels, "reached": st.reached,
                "edges": st.edges}
    if op == "worklist":
        s["wl"].run_device(s["levels"])
        return s["levels"]
    if op == "spmv":
        s["m"].spmv_device(s["x"], s["y"])
        return s["y"]
    with ab.Graph(s["csr"], s["flags"]) as g:
        g.sell_build()
        if s["form"] == "ms":
            out, st = g.msbfs64(s["roots"], out=s["out"])
            return {"levels": out, "reached": st.reached, "edges": st.edges}
        level, parent, st = g.bfs(int(s["roots"][0]))
        return {"level": level, "parent": parent, "reached": st.reached, "edges": st.edges}


def _entries(case):
    """Stored entries, about: duplicates removed, both directions kept."""
    n, ef = case["n"], case["ef"]
    if case["graph"] == "grid":
        return 3.6 * n
    return (1.9 if case["graph"] == "rmat" else 2.0) * n * ef


def work(case):
    """A search cannot do without one source id per reached vertex and its
    outputs; a batched one reads every column once; the fp64 product reads 12
    bytes per entry and reads and writes its vectors; from host memory, the
    CSR goes to the device and the outputs come back."""
    op = case["op"]
    if op == "worklist":
        span = range(case["lo"], case["hi"] + 1)
        n = sum(1 << s for s in span) * case["graphs"] / len(span)
        return {"bytes": n * (4 + 4 * case["roots"]), "flops": 0}
    n, nnz = case["n"], _entries(case)
    if op == "bfs":
        return {"bytes": 12 * n, "flops": 0}
    if op == "ms":
        return {"bytes": 4 * nnz + 256 * n, "flops": 0}
    if op == "spmv":
        return {"bytes": 12 * nnz + 24 * n, "flops": 2 * nnz}
    return {"bytes": 4 * nnz + 8 * n + (256 if case["form"] == "ms" else 8) * n, "flops": 0}


def exact(case, seed):
    """The fp64 product by torch's segment reduction; searches return whole
    numbers, which have no error to measure."""
    if case["op"] != "spmv":
        return None
    rp, col, val, x = _matrix(case, seed)
    return torch.segment_reduce(val * x[col.long()], "sum", offsets=rp, initial=0.0)
