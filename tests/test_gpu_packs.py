"""Packs (several small heads per warp; graphs with 8 vertices and 16 edges for each
of the GPU's 4,736 warps) against the oracle: groups cut by large heads, empty heads, ragged ends, the linear-probing fallback, the id limit, and
their credits per vertex, per edge, per graph and per shard."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import xxtric_b200 as xt
    with xt.Context(0) as c:
        yield c


def graph(kind):
    rng = np.random.default_rng(5)
    if kind == "ring":  # two triangles a vertex, every head alike
        n = 100003
        i = np.arange(n)
        return n, np.concatenate([i, i]), np.concatenate([(i + 1) % n, (i + 2) % n])
    if kind == "gaps":  # triangles between runs of vertices without edges
        n = 500003
        v = np.sort(rng.choice(n // 3, 60000, replace=False)) * 3
        return n, np.concatenate([v, v, v + 1]), np.concatenate([v + 1, v + 2, v + 2])
    if kind == "er":
        n, m = 40017, 200011
        return n, rng.integers(0, n, m), rng.integers(0, n, m)
    if kind == "mixed":  # small heads beside some with hundreds of members
        n = 40001
        a, b = np.triu_indices(700, 1)
        keep = rng.random(len(a)) < 0.5
        m = rng.integers(0, n, (2, 200000))
        p = rng.permutation(n)
        return n, p[np.concatenate([a[keep], m[0]])], p[np.concatenate([b[keep], m[1]])]
    raise ValueError(kind)


@pytest.mark.parametrize("kind", ["ring", "gaps", "er", "mixed"])
@pytest.mark.parametrize("orient", [0, 1])
def test_packs_match_the_oracle(ctx, kind, orient):
    nv, src, dst = graph(kind)
    off, tails = oracle.canon_csr(nv, src.astype(np.int64), dst.astype(np.int64))
    want, pv = oracle.count_merge(off, tails, per_vertex=True)
    sup = oracle.edge_support(off, tails)
    g = ctx.graph_from_edges(nv, src.astype(np.int32), dst.astype(np.int32), orient)
    for iters in (-1, 0, 1):  # 0 and 1: nearly every set falls back to linear probing
        g.debug_cuckoo_iters(iters)
        assert g.count() == want
    total, each = g.count(per_vertex=True)
    assert total == want
    np.testing.assert_array_equal(each, pv)
    a, b, s = g.edge_support()
    u = np.repeat(np.arange(nv), np.diff(off))
    up = u < tails
    order, order_o = np.lexsort((b, a)), np.lexsort((tails[up], u[up]))
    np.testing.assert_array_equal(s[order], sup[up][order_o])
    g.free()


def test_packs_credit_graphs_and_shards(ctx):
    import torch
    graphs = [graph(k) for k in ("ring", "er", "gaps", "ring", "mixed")]
    voff = np.concatenate([[0], np.cumsum([g[0] for g in graphs])])
    eoff = np.concatenate([[0], np.cumsum([len(g[1]) for g in graphs])])
    src = np.concatenate([g[1] for g in graphs]).astype(np.int32)
    dst = np.concatenate([g[2] for g in graphs]).astype(np.int32)
    want = [oracle.count_merge(*oracle.canon_csr(n, s.astype(np.int64), d.astype(np.int64))) for n, s, d in graphs]
    b = ctx.graph_from_batch(voff, eoff, src, dst)
    for iters in (-1, 0):
        b.debug_cuckoo_iters(iters)
        total, per = b.count_groups()
        assert total == sum(want) and per.tolist() == want
    part = torch.zeros(1, dtype=torch.int64, device="cuda")
    got = 0
    for i in range(5):
        b.count_shard_async(i, 5, part)
        ctx.synchronize()
        got += int(part)
    assert got == sum(want)
    b.free()


@pytest.mark.parametrize("nv", [(1 << 26) - 2, (1 << 26) - 1, (1 << 26) + 5])
def test_ids_at_the_pack_limit(ctx, nv):
    # triangles at both ends of the ids; past the limit the heads run one by one
    v = np.concatenate([np.arange(0, 90000, 3), np.arange(nv - 90000, nv - 2, 3)])
    src = np.concatenate([v, v, v + 1]).astype(np.int32)
    dst = np.concatenate([v + 1, v + 2, v + 2]).astype(np.int32)
    for orient in (0, 1):
        g = ctx.graph_from_edges(nv, src, dst, orient)
        assert g.count() == len(v)
        g.free()


@pytest.mark.parametrize("orient", [0, 1])
@pytest.mark.parametrize("span", [0, 40000])
def test_long_warp_tasks_match_the_oracle(ctx, span, orient):
    """Heads of 250 members and up to 32,000 candidates, their members' ids
    within a warp's bitmap or (span) beyond it, some with many short records."""
    rng = np.random.default_rng(3)
    n, k = 70000, 500
    hub = rng.permutation(k) * (1 + span // k)  # the ids of a dense part
    a, b = np.triu_indices(k, 1)
    keep = rng.random(len(a)) < 0.9
    m = rng.integers(0, n, (2, 300000))
    f = rng.integers(0, n, 60000)  # vertices with two neighbours in the dense part
    h = rng.integers(0, k, (2, 60000))
    src = np.concatenate([hub[a[keep]], m[0], f, f])
    dst = np.concatenate([hub[b[keep]], m[1], hub[h[0]], hub[h[1]]])
    off, tails = oracle.canon_csr(n, src.astype(np.int64), dst.astype(np.int64))
    want, pv = oracle.count_merge(off, tails, per_vertex=True)
    sup = oracle.edge_support(off, tails)
    g = ctx.graph_from_edges(n, src.astype(np.int32), dst.astype(np.int32), orient)
    for work in (0, 1 << 20, 1):  # automatic; every head of 256 members on a warp; on CTAs
        g.set_tuning(0, work, 0)
        assert g.count() == want
        total, each = g.count(per_vertex=True)
        assert total == want
        np.testing.assert_array_equal(each, pv)
    g.set_tuning(0, 0, 0)
    u = np.repeat(np.arange(n), np.diff(off))
    up = u < tails
    a, b, s = g.edge_support()
    np.testing.assert_array_equal(s[np.lexsort((b, a))], sup[up][np.lexsort((tails[up], u[up]))])
    g.free()


@pytest.mark.parametrize("kind", ["ring", "gaps", "er", "mixed"])
def test_pack_credits_from_both_tables(ctx, kind):
    """Per-vertex and per-edge counts of packs whose sets are cuckoo tables (the
    default), and where some (1) or nearly all (0) fall back to linear probing."""
    nv, src, dst = graph(kind)
    off, tails = oracle.canon_csr(nv, src.astype(np.int64), dst.astype(np.int64))
    want, pv = oracle.count_merge(off, tails, per_vertex=True)
    sup = oracle.edge_support(off, tails)
    u = np.repeat(np.arange(nv), np.diff(off))
    up = u < tails
    sup = sup[up][np.lexsort((tails[up], u[up]))]
    g = ctx.graph_from_edges(nv, src.astype(np.int32), dst.astype(np.int32))
    for iters in (-1, 1, 0):
        g.debug_cuckoo_iters(iters)
        total, each = g.count(per_vertex=True)
        assert total == want
        np.testing.assert_array_equal(each, pv)
        a, b, s = g.edge_support()
        np.testing.assert_array_equal(s[np.lexsort((b, a))], sup)
    g.free()


@pytest.mark.parametrize("orient", [0, 1])
@pytest.mark.parametrize("ng", [3, 256, 257])
def test_packs_credit_few_and_many_graphs(ctx, ng, orient):
    """Batches of 3 to 257 rings (as many triangles as vertices), whose heads are
    credited to their graphs together or one by one."""
    n = 60000 // ng + np.arange(ng) % 5
    voff = np.concatenate([[0], np.cumsum(n)])
    i = [np.arange(k) for k in n]
    src = np.concatenate([np.concatenate([a, a]) for a in i]).astype(np.int32)
    dst = np.concatenate([np.concatenate([(a + 1) % k, (a + 2) % k]) for a, k in zip(i, n)]).astype(np.int32)
    b = ctx.graph_from_batch(voff, 2 * voff, src, dst, orient)
    total, per = b.count_groups()
    assert total == n.sum() and per.tolist() == n.tolist()
    b.free()
