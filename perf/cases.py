"""The workloads this framework's speed is judged by, as calls of its public API.

A case is a dict of plain values. ``prepare`` makes what a program holds before
the call (inputs on the GPU, resident graph handles), ``run`` is one pass
through the public entry points, ``exact`` the same result in 64 bits without
this package, ``work`` the bytes and operations one pass cannot do without.

Kinds:

* ``solve``     PageRank on a resident graph (``Graph.page_rank``)
* ``seed``      personalised PageRank from one seed (``Graph.ppr``)
* ``drop_in``   the reference's one-shot call on host arrays (``page_rank``)
* ``seeds``     k personalised vectors in one batch (``Graph.ppr_batched``)
* ``teleports`` k teleport vectors on a weighted graph
  (``Graph.weighted_page_rank_batched``)
* ``ragged``    many independent graphs in one batch (``GraphBatch.page_rank``)
* ``gradient``  weighted PageRank and its implicit adjoint, as a training step
* ``build``     a CSR from an edge list on the device (``construct.csr_from_edges``)
* ``spmv``      one weighted sparse matrix-vector product (``Graph.spmv``)

Graphs are RMAT samples (a/b/c/d = .57/.19/.19/.05, symmetrised, deduplicated;
ids modulo n where n is no power of two) or 4-neighbour grids. The seed turns
the vertex ids round by an offset of its own, so every input differs from seed
to seed while a case keeps its size.
"""
import math

import numpy as np
import torch

import nwgraph_b200
from nwgraph_b200 import construct

DAMPING = 0.85


def listed():
    return [
        # A graph of a few thousand entries (an organisation, a test matrix): latency and launches are all of it.
        {"name": "solve_rmat10", "kind": "solve", "graph": "rmat", "n": 1 << 10, "edge_factor": 16, "threshold": 0.0,
         "max_iters": 20},
        # The reference driver's call (threshold 1e-4, at most 20 sweeps) on a graph that stays in L2.
        {"name": "solve_rmat16", "kind": "solve", "graph": "rmat", "n": 1 << 16, "edge_factor": 16, "threshold": 1e-4,
         "max_iters": 20},
        # Low degree, no hubs, many sweeps: road and mesh graphs.
        {"name": "solve_grid1m", "kind": "solve", "graph": "grid", "n": 1000000, "edge_factor": 2, "threshold": 1e-6,
         "max_iters": 200},
        # The headline: 5.2e8 entries, 20 fixed sweeps.
        {"name": "solve_rmat24", "kind": "solve", "graph": "rmat", "n": 1 << 24, "edge_factor": 16, "threshold": 0.0,
         "max_iters": 20},
        # One recommendation query: a single personalised vector.
        {"name": "seed_rmat20", "kind": "seed", "graph": "rmat", "n": 1 << 20, "edge_factor": 16, "threshold": 1e-6,
         "max_iters": 100},
        # A caller of the reference that switches over: host CSR in, host ranks out, nothing resident.
        {"name": "drop_in_rmat18", "kind": "drop_in", "graph": "rmat", "n": 1 << 18, "edge_factor": 16,
         "threshold": 1e-4, "max_iters": 20},
        # 64 personalised vectors of a 4M-vertex graph at once.
        {"name": "seeds_rmat22_k64", "kind": "seeds", "graph": "rmat", "n": 1 << 22, "edge_factor": 16, "k": 64,
         "threshold": 1e-6, "max_iters": 100},
        # 16 topic vectors on a weighted graph.
        {"name": "teleports_rmat20_k16", "kind": "teleports", "graph": "rmat", "n": 1 << 20, "edge_factor": 16, "k": 16,
         "threshold": 1e-6, "max_iters": 300},
        # Hundreds of unrelated graphs of 1e3 to 1e6 vertices, half RMAT, half grids.
        {"name": "ragged_256", "kind": "ragged", "graphs": 256, "max_n": 1000000, "threshold": 1e-6, "max_iters": 200},
        # A training step: ranks, then the gradients of every edge weight and of the teleport vector.
        {"name": "gradient_rmat20", "kind": "gradient", "graph": "rmat", "n": 1 << 20, "edge_factor": 16,
         "threshold": 1e-6, "max_iters": 1000},
        # An edge list to a clean symmetric CSR.
        {"name": "build_rmat20", "kind": "build", "graph": "rmat", "n": 1 << 20, "edge_factor": 16},
        # One sparse product inside a caller's own iteration.
        {"name": "spmv_rmat20", "kind": "spmv", "graph": "rmat", "n": 1 << 20, "edge_factor": 16},
    ]


def _log_size(rng, low, high):
    """A size between low and high, even over its logarithm; odd and ragged ones most of the time."""
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(["solve", "solve", "seed", "drop_in", "seeds", "seeds", "teleports", "ragged", "gradient", "build",
                       "spmv"])
    if kind == "ragged":
        return {"kind": kind, "graphs": _log_size(rng, 16, 256), "max_n": _log_size(rng, 10000, 1000000),
                "threshold": 1e-6, "max_iters": 200}
    top = {"solve": 24, "seed": 22, "drop_in": 20, "seeds": 22, "teleports": 20, "gradient": 20, "build": 22, "spmv": 22}
    case = {"kind": kind, "graph": "rmat", "edge_factor": rng.randint(8, 32)}
    case["n"] = _log_size(rng, 1 << 9, (1 << top[kind]) * 16 // max(16, case["edge_factor"]))
    if kind in ("solve", "seed", "drop_in") and rng.random() < 0.25:
        case.update(graph="grid", edge_factor=2, n=min(case["n"], 1000000))
    if kind in ("solve", "drop_in"):
        fixed = rng.random() < 0.4
        case.update(threshold=0.0 if fixed else rng.choice([1e-4, 1e-6]), max_iters=20)
    elif kind == "seed":
        case.update(threshold=1e-6, max_iters=100)
    elif kind in ("seeds", "teleports"):
        case.update(k=_log_size(rng, 1, 128 if kind == "seeds" else 64), threshold=1e-6, max_iters=100)
        case["n"] = max(512, min(case["n"], (1 << (28 if kind == "seeds" else 24)) // case["k"]))
    elif kind == "gradient":
        case.update(threshold=1e-6, max_iters=1000)
    return case


# ---------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------
def _turned(src, dst, n, seed):
    """The edges with every id moved on by an offset made from the seed, modulo n."""
    by = (2654435761 * (seed + 1)) % n
    return [torch.where(x >= n - by, x - (n - by), x + by) for x in (src, dst)]


def _edges(case, seed, graph_seed=42):
    n = case["n"]
    src, dst = construct.rmat_edges(max(1, math.ceil(math.log2(n))), case["edge_factor"] * n, seed=graph_seed, n=n)
    return _turned(src, dst, n, seed)


def _grid(n, seed):
    side = math.isqrt(n)
    src, dst = _turned(*construct.grid_edges(side), side * side, seed)
    return construct.csr_from_edges(src, dst, side * side, construct.UNDIRECTED)


def _graph(case, seed):
    """(row_ptr, col, degrees) as int32 CUDA tensors."""
    if case["graph"] == "grid":
        return _grid(case["n"], seed)
    src, dst = _edges(case, seed)
    return construct.csr_from_edges(src, dst, case["n"], construct.SIMPLE_UNDIRECTED)


def _random(seed):
    return torch.Generator(device="cuda").manual_seed(7919 + seed)


def _weights(nnz, seed):
    w = torch.rand(nnz, generator=_random(seed), device="cuda", dtype=torch.float32)
    return w.mul_(0.9).add_(0.1)


def _teleports(n, k, seed):
    t = torch.rand((n, k), generator=_random(seed + 1), device="cuda", dtype=torch.float64)
    return (t / t.sum(dim=0, keepdim=True)).float()


def _sources(deg, k, seed):
    """k vertices drawn evenly among those with an edge."""
    some = torch.nonzero(deg > 0).flatten()
    at = np.random.default_rng(seed).integers(0, some.numel(), size=k)
    return some[torch.from_numpy(at).to(some.device)].cpu().numpy().astype(np.uint32)


def _loss(n, seed):
    return torch.randn(n, generator=_random(seed + 2), device="cuda", dtype=torch.float32)


def _ragged(case, seed):
    """Vertex counts log-uniform in [1e3, max_n]; even graphs RMAT with edge factors of 8 to 32, odd ones grids."""
    ns, factors = construct.ragged_sizes(case["graphs"], case["max_n"], 11)
    parts, degrees = [], []
    for g, (n, ef) in enumerate(zip(ns.tolist(), factors.tolist())):
        if g % 2:
            rp, col, deg = _grid(n, seed + g)
        else:
            src, dst = _edges({"n": n, "edge_factor": ef}, seed + g, 11 + g)
            rp, col, deg = construct.csr_from_edges(src, dst, n, construct.SIMPLE_UNDIRECTED)
        parts.append((rp, col))
        degrees.append(deg)
    return parts, degrees


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case}
    if kind == "ragged":
        parts, degs = _ragged(case, seed)
        s["batch"], s["deg"] = construct.batch_from_device_csrs(parts, degs)
        s["out"] = torch.empty(s["batch"].n, dtype=torch.float32, device="cuda")
    elif kind == "build":
        s["src"], s["dst"] = _edges(case, seed)
    else:
        rp, col, deg = _graph(case, seed)
        n = rp.numel() - 1
        s.update(deg=deg, n=n)
        if kind == "drop_in":
            host = [t.cpu().numpy().view(np.uint32) for t in (rp, col, deg)]
            s["csr"], s["deg"] = nwgraph_b200.graphs.CSR(host[0], host[1]), host[2]
            s["out"] = np.empty(n, np.float32)
        elif kind in ("solve", "seed", "seeds"):
            s["graph"] = nwgraph_b200.Graph(rp, col)
            s["out"] = torch.empty(n * case.get("k", 1), dtype=torch.float32, device="cuda")
            if kind != "solve":
                s["seeds"] = _sources(deg, case.get("k", 1), seed)
        else:
            s["graph"] = nwgraph_b200.Graph(rp, col, weights=_weights(col.numel(), seed))
            if kind == "teleports":
                s["t"] = _teleports(n, case["k"], seed)
                s["out"] = torch.empty((n, case["k"]), dtype=torch.float32, device="cuda")
            elif kind == "spmv":
                s["x"] = _loss(n, seed)
                s["out"] = torch.empty(n, dtype=torch.float32, device="cuda")
            else:
                s["c"] = _loss(n, seed)
                s["limit"] = 1e-6 * float(s["c"].abs().sum())
                s["out"] = torch.empty(n, dtype=torch.float32, device="cuda")
                s["dw"] = torch.empty(col.numel(), dtype=torch.float32, device="cuda")
                s["dt"] = torch.empty(n, dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    return s


# ---------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------
def run(s):
    case = s["case"]
    kind = case["kind"]
    stop = (DAMPING, case.get("threshold"), case.get("max_iters"))
    if kind == "solve":
        st = s["graph"].page_rank(s["deg"], s["out"], *stop)
        return {"ranks": s["out"], "sweeps": st.iterations}
    if kind == "seed":
        st = s["graph"].ppr(s["deg"], int(s["seeds"][0]), s["out"], *stop)
        return {"ranks": s["out"], "sweeps": st.iterations}
    if kind == "drop_in":
        nwgraph_b200.page_rank(s["csr"], s["deg"], s["out"], *stop)
        return {"ranks": s["out"]}
    if kind == "seeds":
        st = s["graph"].ppr_batched(s["deg"], s["seeds"], s["out"], *stop)
        return {"ranks": s["out"], "sweeps": st.col_iterations}
    if kind == "teleports":
        st = s["graph"].weighted_page_rank_batched(s["t"], s["out"], *stop)
        return {"ranks": s["out"], "sweeps": st.col_iterations}
    if kind == "ragged":
        st = s["batch"].page_rank(s["deg"], s["out"], *stop)
        return {"ranks": s["out"], "sweeps": st.graph_iterations}
    if kind == "gradient":
        s["graph"].weighted_page_rank(None, s["out"], *stop)
        s["graph"].page_rank_vjp(s["out"], s["c"], s["dw"], s["dt"], DAMPING, s["limit"], case["max_iters"])
        return {"ranks": s["out"], "dw": s["dw"], "dt": s["dt"]}
    if kind == "spmv":
        s["graph"].spmv(s["x"], s["out"])
        return {"y": s["out"]}
    rp, col, deg = construct.csr_from_edges(s["src"], s["dst"], case["n"], construct.SIMPLE_UNDIRECTED)
    return {"row_ptr": rp, "col": col, "degrees": deg}


# ---------------------------------------------------------------------------
# The same in 64 bits
# ---------------------------------------------------------------------------
def _matrix(rp, col, values=None):
    n = rp.numel() - 1
    if values is None:
        values = torch.ones(col.numel(), dtype=torch.float64, device=rp.device)
    return torch.sparse_csr_tensor(rp, col, values, size=(n, n), check_invariants=False)


def _fixed_point(A, out, start, base, threshold, max_iters):
    """x' = base + d A (x / out), each column until the sweep that changes it by less than the threshold in L1."""
    x = start.clone()
    live = torch.ones(x.shape[1], dtype=torch.bool, device=x.device)
    scale = torch.where(out > 0, 1.0 / out, torch.zeros_like(out))[:, None]
    for _ in range(max_iters):
        y = base + DAMPING * (A @ (x * scale))
        change = (y - x).abs().sum(dim=0)
        x = torch.where(live, y, x)
        live = live & ~(change < float(np.float32(threshold)))
        if not bool(live.any()):
            break
    return x


def _exact_ranks(rp, col, deg, threshold, max_iters):
    n = rp.numel() - 1
    x = torch.full((n, 1), 1.0 / n, dtype=torch.float64, device=rp.device)
    return _fixed_point(_matrix(rp, col), deg.double(), x, (1.0 - DAMPING) / n, threshold, max_iters)[:, 0]


def exact(case, seed):
    kind = case["kind"]
    if kind == "build":
        return None  # whole numbers only
    if kind == "ragged":
        parts, degs = _ragged(case, seed)
        ranks = [_exact_ranks(rp, col, deg, case["threshold"], case["max_iters"]) for (rp, col), deg in zip(parts, degs)]
        return {"ranks": torch.cat(ranks), "sweeps": None}
    rp, col, deg = _graph(case, seed)
    n = rp.numel() - 1
    if kind in ("solve", "drop_in"):
        ranks = _exact_ranks(rp, col, deg, case["threshold"], case["max_iters"])
        return {"ranks": ranks, "sweeps": None} if kind == "solve" else {"ranks": ranks.cpu().numpy()}
    if kind in ("seed", "seeds"):
        k = case.get("k", 1)
        e = torch.zeros((n, k), dtype=torch.float64, device=rp.device)
        at = torch.from_numpy(_sources(deg, k, seed).astype(np.int64)).to(rp.device)
        e[at, torch.arange(k, device=rp.device)] = 1.0
        x = _fixed_point(_matrix(rp, col), deg.double(), e, (1.0 - DAMPING) * e, case["threshold"], case["max_iters"])
        return {"ranks": x.reshape(-1), "sweeps": None}
    w = _weights(col.numel(), seed).double()
    A = _matrix(rp, col, w)
    if kind == "spmv":
        return {"y": A @ _loss(n, seed).double()}
    out = torch.zeros(n, dtype=torch.float64, device=rp.device).index_add_(0, col.long(), w)
    if kind == "teleports":
        t = _teleports(n, case["k"], seed).double()
        return {"ranks": _fixed_point(A, out, t, (1.0 - DAMPING) * t, case["threshold"], case["max_iters"]),
                "sweeps": None}
    t = torch.full((n, 1), 1.0 / n, dtype=torch.float64, device=rp.device)
    r = _fixed_point(A, out, t, (1.0 - DAMPING) * t, case["threshold"], case["max_iters"])[:, 0]
    # l = c + d P^T l with P = A / out; the graph's pattern is symmetric, so A^T has A's rows with other weights
    rows = torch.repeat_interleave(torch.arange(n, device=rp.device), rp.diff().long())
    order = torch.sort(col.long() * n + rows).indices
    At = _matrix(rp, rows[order].int(), w[order])
    scale = torch.where(out > 0, 1.0 / out, torch.zeros_like(out))
    c = _loss(n, seed).double()
    adj = c.clone()
    for _ in range(400):
        new = c + DAMPING * scale * (At @ adj)
        change = float((new - adj).abs().max())
        adj = new
        if change < 1e-13:
            break
    # dL/dw of the entry (row i, column j): d r_j / s_j (l_i - q_j), q_j = (A^T l)_j / s_j
    f, q = DAMPING * r * scale, scale * (At @ adj)
    dw = f[col.long()] * (adj[rows] - q[col.long()])
    return {"ranks": r, "dw": dw, "dt": (1.0 - DAMPING) * adj}


# ---------------------------------------------------------------------------
# What one pass cannot do without
# ---------------------------------------------------------------------------
def _entries(case):
    """About how many entries the case's graph has (repeats and self-loops dropped: 13% at 2^16 vertices, 3% at 2^24)."""
    n, ef = case["n"], case["edge_factor"]
    if case["graph"] == "grid":
        side = math.isqrt(n)
        return 4 * side * (side - 1)
    lost = 0.133 * 2.0 ** (-0.27 * (math.log2(n) - 16.0)) * (ef / 16.0) ** 0.5
    return int(2 * ef * n * (1.0 - min(0.8, lost)))


def work(case):
    """Per sweep: column ids, row pointers and entry weights once, every n-vector read or written once; a sweep count
    typical of the stopping rule where it has one. Flops: one addition per entry and vector (and a product where the
    entries are weighted)."""
    kind = case["kind"]
    if kind == "ragged":
        low, high = 1e3, case["max_n"]
        n = case["graphs"] * (high - low) / math.log(high / low)
        nnz = n * 0.5 * (4.0 + 36.0)
        return {"bytes": 22 * (4.0 * nnz + 24.0 * n), "flops": 22 * nnz}
    nnz, n = float(_entries(case)), float(case["n"])
    if kind == "build":
        m = case["edge_factor"] * n
        return {"bytes": 8.0 * m + 4.0 * nnz + 8.0 * n, "flops": 0.0}
    if kind == "spmv":
        return {"bytes": 8.0 * nnz + 12.0 * n, "flops": 2.0 * nnz}
    if kind == "gradient":
        # 17 forward sweeps, 21 applications of the adjoint, one pass that writes dL/dw
        return {"bytes": 38 * (8.0 * nnz + 28.0 * n) + 8.0 * nnz + 16.0 * n, "flops": 38 * 2.0 * nnz + 2.0 * nnz}
    k = case.get("k", 1)
    if kind == "teleports":
        sweeps = 30
        return {"bytes": sweeps * (8.0 * nnz + 8.0 * n + 20.0 * k * n), "flops": sweeps * 2.0 * nnz * k}
    sweeps = case["max_iters"]
    if case["threshold"] > 0:
        sweeps = min(sweeps, 7 if case["threshold"] >= 1e-4 else 14)
        if case["graph"] == "grid":
            sweeps = min(case["max_iters"], 20)
    total = sweeps * (4.0 * nnz + 8.0 * n + 16.0 * k * n)
    if kind == "drop_in":
        total += 4.0 * nnz + 12.0 * n
    return {"bytes": total, "flops": sweeps * nnz * k}
