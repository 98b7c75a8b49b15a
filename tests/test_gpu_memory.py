"""Memory that cannot be had for the dense core: the build goes on without it,
per-vertex and per-edge counts without its operands, all exact."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    import xxtric_b200 as xt
    with xt.Context(0) as c:
        yield c


def wide_core(n_core=600, n_band=20000, per_row=160):
    """A dense core below a band of rows that reach into it: some 160 row blocks of
    three column steps."""
    rng = np.random.default_rng(17)
    a, b = np.triu_indices(n_core, 1)
    keep = rng.random(len(a)) < 0.8
    band = np.repeat(np.arange(n_core, n_core + n_band), per_row)
    t = rng.integers(n_core, n_core + n_band, (2, 30000))
    src = np.concatenate([a[keep], band, t[0]])
    dst = np.concatenate([b[keep], rng.integers(0, n_core, len(band)), t[1]])
    n = n_core + n_band
    p = rng.permutation(n)
    return n, p[src].astype(np.int32), p[dst].astype(np.int32)


class Want:
    def __init__(self):
        self.nv, self.src, self.dst = wide_core()
        off, tails = oracle.canon_csr(self.nv, self.src.astype(np.int64), self.dst.astype(np.int64))
        self.total, self.pv = oracle.count_merge(off, tails, per_vertex=True)
        u = np.repeat(np.arange(self.nv), np.diff(off))
        up = u < tails
        self.by_position = None
        self.sup = oracle.edge_support(off, tails)[up][np.lexsort((tails[up], u[up]))]

    def build(self, ctx):
        return ctx.graph_from_edges(self.nv, self.src, self.dst)

    def check_vertices(self, g):
        total, each = g.count(per_vertex=True)
        assert total == self.total
        np.testing.assert_array_equal(each, self.pv)

    def check_edges(self, g):
        total, sup = g.count_edges()
        assert total == self.total
        if self.by_position is None:  # the supports in the graph's own order, the same for every build
            off, col = g.csr()
            p = g.perm().astype(np.int64)
            a, b = p[np.repeat(np.arange(self.nv), np.diff(off))], p[col]
            self.by_position = np.empty_like(self.sup)
            self.by_position[np.lexsort((np.maximum(a, b), np.minimum(a, b)))] = self.sup
        np.testing.assert_array_equal(sup, self.by_position)


@pytest.fixture(scope="module")
def want():
    return Want()


def count_launches(ctx, g, want):
    before = ctx.launches
    assert g.count() == want.total
    return ctx.launches - before


def test_a_build_goes_on_without_its_core(ctx, want):
    import xxtric_b200 as xt
    g = want.build(ctx)
    full = count_launches(ctx, g, want)
    g.free()
    held = ctx.mem_stats()[0]
    dropped, k = 0, 0
    while True:
        k += 1
        assert k < 200
        ctx.fail_alloc_after(k)
        before = ctx.mem_stats()[0]
        try:
            g = want.build(ctx)
        except xt.XtError as err:
            assert err.status == xt.XT_ERR_OOM
            assert ctx.mem_stats()[0] == before
            continue
        finally:
            ctx.fail_alloc_after(0)
        if count_launches(ctx, g, want) == full:  # no allocation failed
            g.free()
            break
        dropped += 1
        want.check_vertices(g)
        want.check_edges(g)
        g.free()
        assert ctx.mem_stats()[0] == held
    # the tables of its row blocks, their sums, the tiles, the entries before them, the items
    assert dropped == 5


def test_a_core_does_not_raise_the_builds_peak(ctx, want):
    def peak():
        ctx.synchronize()
        before = ctx.mem_stats(reset_peak=True)[0]
        g = want.build(ctx)
        p = ctx.mem_stats()[1] - before
        n = count_launches(ctx, g, want)
        g.free()
        return p, n

    with_core, launches = peak()
    for k in range(1, 200):  # the first allocation whose failure drops the core
        ctx.fail_alloc_after(k)
        try:
            without, n = peak()
            break
        except Exception:
            continue
        finally:
            ctx.fail_alloc_after(0)
    assert n < launches
    assert with_core <= without + (64 << 10)  # the row blocks' tables


@pytest.mark.parametrize("mode", ["vertices", "edges"])
def test_counts_without_operands(ctx, want, mode):
    """The k-th allocation of the first such count fails, on a graph of its own."""
    import xxtric_b200 as xt
    call = want.check_vertices if mode == "vertices" else want.check_edges
    # per vertex: the result, the records' tails, the counts; then S and the rows' sums
    # per edge: the result, the counts; then S, the lists, the transposes and the rows' sums
    needed, core = (3, 2) if mode == "vertices" else (2, 4)
    g = want.build(ctx)
    call(g)
    full = ctx.mem_stats()[0]
    g.free()
    for k in range(1, needed + core + 2):
        g = want.build(ctx)
        ctx.fail_alloc_after(k)
        try:
            call(g)
            assert k > needed
        except xt.XtError as err:
            assert k <= needed and err.status == xt.XT_ERR_OOM
        finally:
            ctx.fail_alloc_after(0)
        call(g)  # and with the memory
        assert ctx.mem_stats()[0] == full
        g.free()


@pytest.mark.parametrize("nshards", [2, 3])
def test_shards_with_and_without_operands_add_up(ctx, want, nshards):
    """One shard counts without the operands, the others with them."""
    import torch
    part = torch.zeros(1, dtype=torch.int64, device="cuda")
    g = want.build(ctx)
    m = g.info()["n_edges"]
    want.check_edges(g)
    g.free()
    for alone in range(nshards):
        pv, es, totals = np.zeros(want.nv, np.int64), np.zeros(m, np.int64), np.zeros(2, np.int64)
        for i in range(nshards):
            g = want.build(ctx)
            each = torch.zeros(want.nv, dtype=torch.int64, device="cuda")
            edge = torch.zeros(m, dtype=torch.int64, device="cuda")
            torch.cuda.synchronize()
            g.count_shard_async(i, nshards, part)  # the shards' schedule
            ctx.fail_alloc_after(3 if i == alone else 0)  # the records' tails, the counts, S
            g.count_shard_async(i, nshards, part, each)
            ctx.synchronize()
            totals[0] += int(part)
            ctx.fail_alloc_after(3 if i == alone else 0)  # counts, S, the lists
            g.count_edges_shard_async(i, nshards, part, edge)
            ctx.synchronize()
            ctx.fail_alloc_after(0)
            totals[1] += int(part)
            pv += each.cpu().numpy()
            es += edge.cpu().numpy()
            g.free()
        assert (totals == want.total).all()
        np.testing.assert_array_equal(pv, want.pv)
        np.testing.assert_array_equal(es, want.by_position)


@pytest.mark.parametrize("nshards", [2, 16])
def test_shards_of_every_size_add_up(ctx, want, nshards):
    """Two shards count their part of the core, sixteen stream all their records; the
    same after the schedule has been made anew."""
    import torch
    g = want.build(ctx)
    want.check_edges(g)
    part = torch.zeros(1, dtype=torch.int64, device="cuda")
    each = torch.zeros(want.nv, dtype=torch.int64, device="cuda")
    edge = torch.zeros(len(want.by_position), dtype=torch.int64, device="cuda")
    torch.cuda.synchronize()
    for again in range(2):
        totals, pv, es = np.zeros(3, np.int64), np.zeros(want.nv, np.int64), np.zeros(len(edge), np.int64)
        before = ctx.launches
        for i in range(nshards):
            g.count_shard_async(i, nshards, part)
            ctx.synchronize()
            totals[0] += int(part)
        if again:
            assert (ctx.launches - before == 3 * nshards) == (nshards == 2), "with the core's kernel, or without"
        for i in range(nshards):
            g.count_shard_async(i, nshards, part, each)
            ctx.synchronize()
            totals[1] += int(part)
            pv += each.cpu().numpy()
            g.count_edges_shard_async(i, nshards, part, edge)
            ctx.synchronize()
            totals[2] += int(part)
            es += edge.cpu().numpy()
        assert (totals == want.total).all()
        np.testing.assert_array_equal(pv, want.pv)
        np.testing.assert_array_equal(es, want.by_position)
        want.check_vertices(g)
        if not again:
            g.set_tuning(0, 2048, 0)
            g.set_tuning(0, 0, 0)
            g.count_shard_async(0, nshards, part)  # builds what the next launches do not
            g.count_shard_async(0, nshards, part, each)
            ctx.synchronize()
    g.free()


def test_shards_recorded_before_they_ran(want):
    """Shards whose first count is recorded, and those that run, share the work out
    alike; a recorded one stays right after counts of many other numbers of shards."""
    import torch
    import xxtric_b200 as xt
    stream = torch.cuda.Stream()
    with xt.Context(0) as c:
        c.set_stream(stream.cuda_stream)
        for nshards in (2, 16):
            graphs = [want.build(c) for _ in range(2)]
            part = torch.zeros(2, dtype=torch.int64, device="cuda")
            torch.cuda.synchronize()
            rec = torch.cuda.CUDAGraph()
            with torch.cuda.graph(rec, stream=stream):
                graphs[0].count_shard_async(0, nshards, part[0:1])
            got = 0
            for i in range(1, nshards):  # the others, run on a graph of their own
                graphs[1].count_shard_async(i, nshards, part[1:2])
                c.synchronize()
                got += int(part[1])
            for others in (range(2, 3), range(2, 14)):
                for k in others:
                    graphs[0].count_shard_async(k - 1, k, part[1:2])
                c.synchronize()
                part.zero_()
                torch.cuda.synchronize()
                rec.replay()
                torch.cuda.synchronize()
                assert int(part[0]) + got == want.total
            del rec
            torch.cuda.synchronize()
            for g in graphs:
                g.free()
