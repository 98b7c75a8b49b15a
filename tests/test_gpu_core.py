"""The dense core (blocks of the top ranks counted on the tensor cores) against
the oracle, at the edges of its row blocks (128), column steps (256) and
widths, and beside rows that are streamed."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import xxtric_b200 as xt
    with xt.Context(0) as c:
        yield c


def dense(n, p, rng):
    a, b = np.triu_indices(n, 1)
    keep = rng.random(len(a)) < p
    return a[keep], b[keep]


def graph(kind):
    rng = np.random.default_rng(11)
    if isinstance(kind, int):  # a dense graph of that many vertices
        return kind, *dense(kind, 0.8, rng)
    if kind == "complete":
        return 1700, *np.triu_indices(1700, 1)
    if kind == "core and tail":  # a dense core, a band of rows half in it, and a sparse tail
        n, k = 60000, 1500
        a, b = dense(k, 0.6, rng)
        m = rng.integers(k, 6000, 250000)
        t = rng.integers(0, n, (2, 200000))
        s = np.concatenate([a, m, t[0]])
        d = np.concatenate([b, rng.integers(0, k, len(m)), t[1]])
        p = rng.permutation(n)
        return n, p[s], p[d]
    raise ValueError(kind)


CASES = [1151, 1152, 1153, 1279, 1280, 1281, 1535, 1537, "complete", "core and tail"]


@pytest.mark.parametrize("kind", CASES)
def test_core_counts_match_the_oracle(ctx, kind):
    nv, src, dst = graph(kind)
    off, tails = oracle.canon_csr(nv, src.astype(np.int64), dst.astype(np.int64))
    want, pv = oracle.count_merge(off, tails, per_vertex=True)
    want_sup = oracle.edge_support(off, tails)
    u = np.repeat(np.arange(nv), np.diff(off))
    up = u < tails
    want_sup = want_sup[up]
    g = ctx.graph_from_edges(3, np.array([0, 0, 1], np.int32), np.array([1, 2, 2], np.int32))
    before = ctx.launches
    assert g.count() == 1
    plain = ctx.launches - before  # launches of a count without a core
    g.free()
    for orient in (1, 0):
        g = ctx.graph_from_edges(nv, src.astype(np.int32), dst.astype(np.int32), orient)
        before = ctx.launches
        assert g.count() == want
        if orient == 1 or kind != "core and tail":  # under the id order the permuted core is not at the top
            assert ctx.launches > before + plain, "the core's kernel beside the streaming one"
        total, each = g.count(per_vertex=True)
        assert total == want
        np.testing.assert_array_equal(each, pv)
        a, b, sup = g.edge_support()
        order = np.lexsort((b, a))
        np.testing.assert_array_equal(sup[order], want_sup[np.lexsort((tails[up], u[up]))])
        g.set_tiers(0, 0)
        assert g.count() == want
        g.free()


@pytest.mark.parametrize("nshards", [2, 7])
def test_core_shards_sum_to_the_count(ctx, nshards):
    import torch
    nv, src, dst = graph("core and tail")
    g = ctx.graph_from_edges(nv, src.astype(np.int32), dst.astype(np.int32))
    want, pv = g.count(per_vertex=True)
    total, sup = g.count_edges()
    assert g.count() == total == want
    part = torch.zeros(1, dtype=torch.int64, device="cuda")
    each = torch.zeros(nv, dtype=torch.int64, device="cuda")
    edge = torch.zeros(len(sup), dtype=torch.int64, device="cuda")
    got = np.zeros(3, np.int64)
    pvs, sups = np.zeros_like(pv), np.zeros_like(sup)
    torch.cuda.synchronize()
    for i in range(nshards):
        g.count_shard_async(i, nshards, part)
        ctx.synchronize()
        got[0] += int(part)
        g.count_shard_async(i, nshards, part, each)
        ctx.synchronize()
        got[1] += int(part)
        pvs += each.cpu().numpy()
        g.count_edges_shard_async(i, nshards, part, edge)
        ctx.synchronize()
        got[2] += int(part)
        sups += edge.cpu().numpy()
    assert (got == want).all()
    np.testing.assert_array_equal(pvs, pv)
    np.testing.assert_array_equal(sups, sup)
    g.free()


@pytest.mark.parametrize("first", ["recorded", "run"])
def test_core_counts_recorded_and_replayed(ctx, first):
    """Counts recorded into a CUDA graph and replayed twice, before and after
    the operands of the per-edge product exist."""
    import torch
    import xxtric_b200 as xt
    nv, src, dst = graph("core and tail")
    off, tails = oracle.canon_csr(nv, src.astype(np.int64), dst.astype(np.int64))
    want, pv = oracle.count_merge(off, tails, per_vertex=True)
    stream = torch.cuda.Stream()
    with xt.Context(0) as c:
        c.set_stream(stream.cuda_stream)
        g = c.graph_from_edges(nv, src.astype(np.int32), dst.astype(np.int32))
        m = g.info()["n_edges"]
        each = torch.zeros(nv, dtype=torch.int64, device="cuda")
        edge = torch.zeros(m, dtype=torch.int64, device="cuda")
        total = torch.zeros(3, dtype=torch.int64, device="cuda")
        torch.cuda.synchronize()

        def counts():
            g.count_async(total[0:1])
            g.count_edges_async(total[1:2], edge)
            if first == "run":  # the records' tails, which any graph's per-vertex count keeps, exist by then
                g.count_async(total[2:3], each)

        if first == "run":
            counts()
            c.synchronize()
        rec = torch.cuda.CUDAGraph()
        with torch.cuda.graph(rec, stream=stream):
            counts()
        for _ in range(2):
            total.zero_(), each.zero_(), edge.zero_()
            torch.cuda.synchronize()
            rec.replay()
            torch.cuda.synchronize()
            assert total.tolist()[:2] == [want] * 2
            if first == "run":
                assert int(total[2]) == want
                np.testing.assert_array_equal(each.cpu().numpy(), pv)
            assert int(edge.sum()) == 3 * want
        del rec
        torch.cuda.synchronize()
        assert g.count() == want  # and uncaptured again
        g.capture()
        assert g.count() == g.count_groups()[0] == want
        g.free()


def test_core_allocations_that_fail(ctx):
    """Each allocation of a build and of its counts fails once; the context and
    the graph stay usable and nothing is left behind."""
    import xxtric_b200 as xt
    nv, src, dst = graph(1281)
    src, dst = src.astype(np.int32), dst.astype(np.int32)
    want = oracle.count_merge(*oracle.canon_csr(nv, src.astype(np.int64), dst.astype(np.int64)))

    def until_it_passes(call):
        for k in range(1, 200):
            ctx.fail_alloc_after(k)
            try:
                return call()
            except xt.XtError as err:
                assert err.status == xt.XT_ERR_OOM
            finally:
                ctx.fail_alloc_after(0)
        raise AssertionError("still failing")

    held = ctx.mem_stats()[0]
    g = until_it_passes(lambda: ctx.graph_from_edges(nv, src, dst))
    assert g.count() == want
    assert until_it_passes(g.count_edges)[0] == want
    assert until_it_passes(lambda: g.count(per_vertex=True))[0] == want
    g.free()
    assert ctx.mem_stats()[0] == held


def test_footprint_counts_the_core(ctx):
    """footprint_bytes: every array a count reads, the core's tiles (16 KB each) and
    items (8 bytes) among them."""
    def parts(g, nv):
        i, off = g.info(), g.csr()[0]
        padded = int(((np.diff(off) + 7) // 8 * 8).sum())
        return i["footprint_bytes"] - (16 * (nv + 1) + 8 * nv + 12 * i["n_edges"] + 4 * padded)
    g = ctx.graph_from_edges(3, np.array([0, 0, 1], np.int32), np.array([1, 2, 2], np.int32))
    assert parts(g, 3) == 0
    g.free()
    # 1,280 dense vertices: 10 row blocks, pairs of them of width 1 to 5 column steps, each
    # stored in an even number of chunks
    nv, src, dst = graph(1280)
    g = ctx.graph_from_edges(nv, src.astype(np.int32), dst.astype(np.int32))
    core = parts(g, nv)
    assert core >= 16384 * 2 * 2 * (1 + 2 + 3 + 4 + 5)
    assert core <= 16384 * (2 * 2 * (1 + 2 + 3 + 4 + 5) + 2 * 5 * 128)
    g.free()


def test_supports_of_a_wide_core_sum_to_the_vertices_counts(ctx):
    """R-MAT 2^20, whose core is thousands of positions wide and its products cut into
    many segments: the supports sum to three times the total, and those around each
    vertex to twice its own count (which the oracle's digests check elsewhere)."""
    import torch
    scale = 20
    rows = 16 << scale
    src = torch.empty(rows, dtype=torch.int32, device="cuda")
    dst = torch.empty_like(src)
    torch.cuda.synchronize()
    ctx.gen_rmat(scale, rows, 5, src, dst)
    g = ctx.graph_from_device_edges(1 << scale, rows, src, dst)
    total, each = g.count(per_vertex=True)
    total_e, sup = g.count_edges()
    assert total == total_e == g.count()
    off, col = g.csr()
    p = g.perm()
    a, b = p[np.repeat(np.arange(len(off) - 1), np.diff(off))], p[col]
    n = len(off) - 1
    around = np.bincount(a, sup, n) + np.bincount(b, sup, n)  # whole numbers far below 2^53
    assert int(sup.sum()) == 3 * total
    np.testing.assert_array_equal(around.astype(np.int64), 2 * each)
    g.free()
