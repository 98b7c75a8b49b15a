"""What users of this framework have it do, as cases that can be timed.

Every case is one pass through public entry points of ``xxtric_b200``: a count
of a graph that is resident on the GPU (global, per vertex, per edge), a whole
step from host or device input to the count, or a batch of small graphs.

A case is a dict of plain values:

  op      count       global count of a resident graph (``DeviceGraph.count``)
          vertices    per-vertex counts into device memory (``count_async``)
          edges       per-edge supports into device memory (``count_edges_async``)
          build       host edge list -> build -> count -> free
          csr         host CSR -> ``TriangleCountingSingle`` -> count -> clear
          device      device CSR in the reference's layout -> ``count_device``
          batch       many host graphs -> ``batch_count`` in one call
          generate    random geometric graph generated, built and counted
  family  rmat | er | chunglu | rgg: the graph (op "batch": "mixed", half random
          geometric and half Erdos-Renyi graphs of 256 to 65,535 vertices)
  n       vertices (a power of two for R-MAT and Chung-Lu, whose ids are
          permuted); graphs of the batch for op "batch"
  degree  input rows per vertex (rgg: mean degree, which sets the radius)
  orient  the library's orientation: 1 by degree (the default), 0 by id
"""
import math

import numpy as np
import torch

import xxtric_b200 as xt

_DEVICE = 0
_ctx = None


def _context():
    """One context per process, as a program of a user would hold."""
    global _ctx
    if _ctx is None:
        _ctx = xt.Context(_DEVICE)
    return _ctx


def listed():
    return [
        # A geometric graph of the size the command-line driver's examples use:
        # a count that is launches and latency.
        {"name": "count rgg 65k", "op": "count", "family": "rgg", "n": 65536, "degree": 16.0, "orient": 1},
        # The sample on which the reference's CPU engine is compared.
        {"name": "count rmat 2^18", "op": "count", "family": "rmat", "n": 1 << 18, "degree": 16.0, "orient": 1},
        # An ordinary power-law graph, counted repeatedly.
        {"name": "count rmat 2^22", "op": "count", "family": "rmat", "n": 1 << 22, "degree": 16.0, "orient": 1},
        # The headline benchmark's graph.
        {"name": "count rmat 2^24", "op": "count", "family": "rmat", "n": 1 << 24, "degree": 16.0, "orient": 1},
        # The skewed benchmark graph: a few hubs next to most of the others.
        {"name": "count chunglu 2^22", "op": "count", "family": "chunglu", "n": 1 << 22, "degree": 32.0, "orient": 1},
        # Local clustering coefficients: a count for every vertex.
        {"name": "vertices rmat 2^21", "op": "vertices", "family": "rmat", "n": 1 << 21, "degree": 16.0, "orient": 1},
        # k-truss support: a count for every edge.
        {"name": "edges rmat 2^20", "op": "edges", "family": "rmat", "n": 1 << 20, "degree": 16.0, "orient": 1},
        # A new graph per step from pinned host memory (the end-to-end metric).
        {"name": "build rmat 2^21", "op": "build", "family": "rmat", "n": 1 << 21, "degree": 16.0, "orient": 1},
        # The reference's engine class on a CSR read from a file.
        {"name": "csr rgg 2^18", "op": "csr", "family": "rgg", "n": 1 << 18, "degree": 24.0, "orient": 1},
        # The reference's kernel launcher on its device CSR.
        {"name": "device rmat 2^20", "op": "device", "family": "rmat", "n": 1 << 20, "degree": 16.0, "orient": 1},
        # Many small graphs in one call.
        {"name": "batch 256", "op": "batch", "family": "mixed", "n": 256, "degree": 0.0, "orient": 1},
        # The command-line driver's -n path.
        {"name": "generate rgg 2^20", "op": "generate", "family": "rgg", "n": 1 << 20, "degree": 16.0, "orient": 1},
    ]


def draw(rng):
    """Another case of the same ranges: sizes log-uniform from thousands of rows
    to the listed cases' largest, both orientations where the input's own order
    is not skewed against the lower ids."""
    op = rng.choice(["count", "count", "count", "count", "vertices", "vertices", "edges", "edges", "build", "build",
                     "csr", "device", "batch", "generate"])
    if op == "batch":
        return {"op": op, "family": "mixed", "n": int(round(2 ** rng.uniform(2, 8))), "degree": 0.0,
                "orient": rng.choice([0, 1, 1])}
    if op == "generate":
        return {"op": op, "family": "rgg", "n": int(2 ** rng.uniform(12, 20)), "degree": round(rng.uniform(6, 32), 2),
                "orient": rng.choice([0, 1, 1])}
    family = rng.choice(["rmat", "rmat", "chunglu", "er", "rgg"])
    degree = round(2 ** rng.uniform(2, 5), 2)
    top = {"count": 27.5, "vertices": 25.0, "edges": 24.0, "build": 25.0, "csr": 22.5, "device": 24.0}[op]
    rows = 2 ** rng.uniform(13, top)  # input rows: n * degree
    orient = rng.choice([0, 1, 1, 1]) if op != "device" else 1  # count_device orients by degree
    if family == "er" or family == "rgg":
        n = max(64, int(rows / degree)) | 1
    else:
        n = 1 << max(8, int(round(math.log2(rows / degree))))
        if family == "chunglu":
            n = min(n, 1 << 22)
        if rows > 2 ** 22:
            orient = 1  # hubs of low ids make the id order's work grow out of these ranges
    if family == "rgg":
        n = min(n, 1 << 22)
    return {"op": op, "family": family, "n": n, "degree": degree, "orient": orient}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _radius(n, degree, seed):
    """The radius of the mean degree; the seed moves it by up to 2%."""
    return math.sqrt(degree / (math.pi * n)) * (1.0 + 0.02 * ((seed * 2654435761) % 1000) / 1000.0)


def _device_rows(case, seed):
    """(n, rows, src, dst): the case's int32 edge rows on the GPU."""
    ctx, n = _context(), case["n"]
    if case["family"] == "rgg":
        m, src, dst = ctx.gen_rgg(n, 1, _radius(n, case["degree"], seed))
        return n, m, src, dst
    rows = int(n * case["degree"])
    if case["family"] == "chunglu":
        cdf, rows = xt.chunglu_cdf(n, 2.1, 2.0 * case["degree"], max(64.0, n / 32.0))
    src = torch.empty(rows, dtype=torch.int32, device="cuda")
    dst = torch.empty_like(src)
    torch.cuda.synchronize()
    if case["family"] == "rmat":
        ctx.gen_rmat(n.bit_length() - 1, rows, seed, src, dst)
    elif case["family"] == "chunglu":
        ctx.gen_chunglu(cdf, rows, seed, src, dst)
    else:
        ctx.gen_er(n, rows, seed, src, dst)
    return n, rows, src, dst


def _symmetric_keys(n, src, dst):
    """Sorted unique keys row * n + tail of the undirected graph, both directions."""
    s, d = src.long(), dst.long()
    keep = s != d
    s, d = s[keep], d[keep]
    return torch.unique(torch.cat([s * n + d, d * n + s]))


def _csr(n, src, dst):
    """The reference's CSR: int64 offsets and tails, rows sorted, symmetric."""
    key = _symmetric_keys(n, src, dst)
    rows = torch.div(key, n, rounding_mode="floor")
    off = torch.zeros(n + 1, dtype=torch.int64, device=key.device)
    off[1:] = torch.cumsum(torch.bincount(rows, minlength=n), 0)
    return off, key - rows * n


def _pinned(t):
    h = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    h.copy_(t)
    return h.numpy()


def _batch_rows(case, seed):
    """A batch's tables and its local-id rows in pinned host memory."""
    ctx = _context()
    spec = xt.batch_spec(case["n"], seed)
    eoff, src, dst = ctx.gen_batch(spec)
    voff = np.zeros(case["n"] + 1, np.int64)
    np.cumsum(spec["n"], out=voff[1:])
    if int(eoff[-1]):
        host = [_pinned(torch.as_tensor(a, device="cuda")) for a in (src, dst)]
    else:
        host = [np.zeros(0, np.int32), np.zeros(0, np.int32)]
    torch.cuda.synchronize()
    src.free()
    dst.free()
    return voff, np.asarray(eoff), host[0], host[1]


def prepare(case, seed):
    ctx, op = _context(), case["op"]
    state = {"op": op, "orient": case["orient"]}
    if op == "generate":
        state.update(n=case["n"], radius=_radius(case["n"], case["degree"], seed))
        return state
    if op == "batch":
        state["batch"] = _batch_rows(case, seed)
        return state
    n, rows, src, dst = _device_rows(case, seed)
    state["n"] = n
    if op in ("count", "vertices", "edges"):
        state["graph"] = ctx.graph_from_device_edges(n, rows, src, dst, case["orient"])
        state["total"] = torch.zeros(1, dtype=torch.int64, device="cuda")
        if op == "vertices":
            state["each"] = torch.zeros(n, dtype=torch.int64, device="cuda")
        elif op == "edges":
            # one entry for each input row: at least as many as distinct edges
            state["each"] = torch.zeros(max(1, rows), dtype=torch.int64, device="cuda")
    elif op == "build":
        state["src"], state["dst"] = _pinned(src), _pinned(dst)
    else:
        off, tails = _csr(n, src, dst)
        if op == "csr":
            state["off"], state["tails"] = _pinned(off), _pinned(tails)
        else:
            state["off"], state["tails"] = off, tails
            state["total"] = torch.zeros(1, dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    return state


def run(state):
    op = state["op"]
    if op == "count":
        return state["graph"].count()
    if op == "vertices":
        state["graph"].count_async(state["total"], state["each"])
        return state["total"], state["each"]
    if op == "edges":
        state["graph"].count_edges_async(state["total"], state["each"])
        return state["total"], state["each"]
    if op == "build":
        g = _context().graph_from_edges(state["n"], state["src"], state["dst"], state["orient"])
        total = g.count()
        g.free()
        return total
    if op == "csr":
        engine = xt.TriangleCountingSingle(state["off"], state["tails"], state["orient"], _DEVICE)
        total = engine.count()
        engine.clear()
        return total
    if op == "device":
        xt.count_device(state["n"], state["off"], state["tails"], state["total"])
        return state["total"]
    if op == "batch":
        return _context().batch_count(*state["batch"], state["orient"])
    g = _context().graph_from_rgg(state["n"], 1, state["radius"], state["orient"])
    total = g.count()
    g.free()
    return total


def work(case):
    """The bytes that a pass has to move: the oriented graph (4 bytes an edge
    and 8 a vertex) or the input in its own layout read once, results written
    once. The comparisons of a count depend on the graph and are not stated."""
    op, n = case["op"], case["n"]
    if op == "batch":
        # means of the batch's distributions: 11,770 vertices, mean degree 26.9, each edge one row
        return {"bytes": n * (11770 * 13.45 * 8 + 8), "flops": 0}
    if op == "generate":
        return {"bytes": n * 16.0, "flops": 0}
    m = n * case["degree"]
    if case["family"] == "rgg":
        m /= 2
    if op == "build":
        return {"bytes": 8 * m + 8, "flops": 0}
    if op in ("csr", "device"):
        return {"bytes": 16 * m + 8 * (n + 1) + 8, "flops": 0}
    out = {"count": 8, "vertices": 8 * n + 8, "edges": 8 * m + 8}[op]
    return {"bytes": 4 * m + 8 * (n + 1) + out, "flops": 0}


# ---------------------------------------------------------------------------
# the counts by plain torch
# ---------------------------------------------------------------------------

_MOST_WEDGES = 1 << 31


def _count_plain(n, src, dst, per_vertex=False):
    """Triangles of the undirected graph by closing every wedge u < v < w of the
    (degree, id) order against the sorted edge keys; None beyond 2^31 wedges."""
    key = _symmetric_keys(n, src, dst)
    a, b = torch.div(key, n, rounding_mode="floor"), key % n
    rank = torch.empty(n, dtype=torch.int64, device=key.device)
    order = torch.sort(torch.bincount(a, minlength=n), stable=True).indices
    rank[order] = torch.arange(n, device=key.device)
    a, b = rank[a], rank[b]
    key = torch.sort(a[a < b] * n + b[a < b]).values
    u, v = torch.div(key, n, rounding_mode="floor"), key % n
    end = torch.cumsum(torch.bincount(u, minlength=n), 0)
    after = end[u] - 1 - torch.arange(len(u), device=key.device)  # columns of u's row behind each edge
    reach = torch.cumsum(after, 0)
    if len(u) == 0 or int(reach[-1]) > _MOST_WEDGES:
        return (None if len(u) else 0), (None if len(u) else torch.zeros(n, dtype=torch.int64))
    total, each = 0, torch.zeros(n, dtype=torch.int64, device=key.device)
    at = 0
    while at < len(u):
        base = int(reach[at - 1]) if at else 0
        to = max(at + 1, int(torch.searchsorted(reach, base + (1 << 26), right=True)))
        e = torch.repeat_interleave(torch.arange(at, to, device=key.device), after[at:to])
        first = (reach - after)[e] - base
        w = v[e + 1 + torch.arange(len(e), device=key.device) - first]
        probe = v[e] * n + w
        i = torch.searchsorted(key, probe).clamp(max=len(key) - 1)
        hit = key[i] == probe
        total += int(hit.sum())
        if per_vertex:
            for x in (u[e], v[e], w):
                each += torch.bincount(x[hit], minlength=n)
        at = to
    return total, each[rank]


def exact(case, seed):
    """The counts of small and middling graphs without this library's counting.
    Supports are listed in the library's own edge order, which this does not
    restate."""
    op = case["op"]
    if op == "batch":
        voff, eoff, src, dst = _batch_rows(case, seed)
        if int(eoff[-1]) > 1 << 22:
            return None
        per = np.zeros(case["n"], np.int64)
        for g in range(case["n"]):
            s, d = (torch.from_numpy(x[eoff[g]:eoff[g + 1]].copy()).cuda() for x in (src, dst))
            per[g] = _count_plain(int(voff[g + 1] - voff[g]), s, d)[0]
        return int(per.sum()), per
    if case["family"] != "rgg" and case["n"] * case["degree"] > 1 << 23:
        return None
    n, _, src, dst = _device_rows(case, seed)
    total, each = _count_plain(n, src, dst, op == "vertices")
    if total is None:
        return None
    if op == "vertices":
        return torch.tensor([total]), each
    if op == "edges":
        return torch.tensor([total]), None
    return torch.tensor([total]) if op == "device" else total
