"""CSR input: rows that are canonical are oriented by counting, without an edge
sort, whether they were promised to be or not; all others take the edge-list
path. Both must leave the same graph."""
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
    """(nv, src, dst) of one shape of rows."""
    rng = np.random.default_rng(7)
    if kind == "one edge":
        return 2, np.array([0]), np.array([1])
    if kind == "empty rows":  # runs of empty rows longer than the linear walk, first and last rows empty
        ids = np.array([13, 14, 40, 41, 900, 2047, 3000])
        a, b = np.meshgrid(ids, ids)
        return 4097, a[a < b], b[a < b]
    if kind == "hub":  # one row over many spans, its neighbours' rows of one or two entries
        n = 5000
        s = np.concatenate([np.zeros(n - 1, np.int64), np.arange(1, n - 1, 2)])
        d = np.concatenate([np.arange(1, n), np.arange(2, n, 2)])
        return n, s, d[:len(s)]
    n, m = {"span": (64, 2 * 128), "span+1": (65, 2 * 128 + 1), "er": (3001, 20011)}[kind]
    if kind == "er":
        return n, rng.integers(0, n, m), rng.integers(0, n, m)
    pairs = rng.permutation(n * (n - 1) // 2)[:m // 2]  # entries: spans of exactly 256, or a little more
    a, b = np.triu_indices(n, 1)
    return n, a[pairs], b[pairs]


@pytest.mark.parametrize("kind", ["one edge", "empty rows", "hub", "span", "span+1", "er"])
@pytest.mark.parametrize("orient", [0, 1])
def test_canonical_rows_give_the_edge_list_graph(ctx, kind, orient):
    nv, src, dst = graph(kind)
    off, tails = oracle.canon_csr(nv, src.astype(np.int64), dst.astype(np.int64))
    want = oracle.count_merge(off, tails)
    u = np.repeat(np.arange(nv), np.diff(off))
    ge = ctx.graph_from_edges(nv, u.astype(np.int32), tails.astype(np.int32), orient)
    for canonical in (True, False):
        g = ctx.graph_from_csr(off, tails, canonical=canonical, orient=orient)
        assert g.count() == want
        for a, b in zip(g.csr(), ge.csr()):
            np.testing.assert_array_equal(a, b)
        np.testing.assert_array_equal(g.perm(), ge.perm())
        assert g.info() == ge.info()
        g.free()
    ge.free()


@pytest.mark.parametrize("drop", ["upper", "lower", "one of each"])
def test_rows_without_their_back_entries_take_the_general_path(ctx, drop):
    import xxtric_b200 as xt
    nv, src, dst = graph("er")
    off, tails = oracle.canon_csr(nv, src.astype(np.int64), dst.astype(np.int64))
    want = oracle.count_merge(off, tails)  # an edge listed from one end is still an edge
    u = np.repeat(np.arange(nv), np.diff(off))
    up, low = np.flatnonzero(u < tails), np.flatnonzero(u > tails)
    gone = {"upper": up[100:101], "lower": low[200:201]}.get(drop)
    if gone is None:  # different edges: as many entries above as below remain
        gone = np.array([up[100], next(e for e in low[500:] if tails[e] != u[up[100]])])
    keep = np.ones(len(tails), bool)
    keep[gone] = False
    off2 = np.concatenate([[0], np.cumsum(np.bincount(u[keep], minlength=nv))])
    with pytest.raises(xt.XtError) as e:
        ctx.graph_from_csr(off2, tails[keep], canonical=True)
    assert e.value.status == xt.XT_ERR_INVALID
    g = ctx.graph_from_csr(off2, tails[keep], canonical=False)
    assert g.count() == want
    g.free()


@pytest.mark.parametrize("before", [1, 70000])
def test_entries_before_the_first_row_are_checked(before):
    """A device CSR whose rows start past entry 0: the entries before them are no
    edges, but an id out of range among them is refused like any other."""
    import torch
    import xxtric_b200 as xt
    off = torch.tensor([0, 2, 4, 6], dtype=torch.int64, device="cuda") + before
    tails = torch.zeros(before + 6, dtype=torch.int64, device="cuda")
    tails[before:] = torch.tensor([1, 2, 0, 2, 0, 1])
    out = torch.zeros(1, dtype=torch.int64, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    xt.count_device(3, off, tails, out, stream=stream)
    assert int(out) == 1
    for rows in (off, torch.full_like(off, before)):  # and where no row has an entry
        for bad in (3, -1):
            tails[before // 2] = bad
            with pytest.raises(xt.XtError) as e:
                xt.count_device(3, rows, tails, out, stream=stream)
            assert e.value.status == xt.XT_ERR_INVALID
