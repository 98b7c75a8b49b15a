"""Bounded device waits that run out: the call reports it, its copies and
products in flight end first, and the next call is exact."""
import contextlib

import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu

NV = 1281  # dense enough for the tensor-core part of the count (its kernels hold the waits)


@contextlib.contextmanager
def waits_give_up():
    import xxtric_b200 as xt
    xt.debug_give_up(True)
    try:
        yield
    finally:
        xt.debug_give_up(False)


def dense_graph():
    rng = np.random.default_rng(3)
    a, b = np.triu_indices(NV, 1)
    keep = rng.random(len(a)) < 0.8
    off, tails = oracle.canon_csr(NV, a[keep], b[keep])
    return off, tails, oracle.count_merge(off, tails, per_vertex=True)


@pytest.fixture(scope="module")
def dense():
    return dense_graph()


def test_core_waits_that_give_up_are_reported(dense):
    """The loader's copies are under way when the other warps leave: the call says
    so, and the next one is exact."""
    import xxtric_b200 as xt
    off, tails, (want, pv) = dense
    with xt.Context(0) as c:
        g = c.graph_from_csr(off, tails)
        for call in (g.count, lambda: g.count(per_vertex=True), g.count_edges):
            for _ in range(3):
                with waits_give_up(), pytest.raises(xt.XtError) as err:
                    call()
                assert err.value.status == xt.XT_ERR_TIMEOUT
                assert g.count() == want
        total, each = g.count(per_vertex=True)
        assert total == want
        np.testing.assert_array_equal(each, pv)
        g.free()


@pytest.mark.parametrize("accumulate", [False, True])
def test_count_device_reports_a_wait_that_ran_out(dense, accumulate):
    import torch
    import xxtric_b200 as xt
    off, tails, (want, _) = dense
    d_off, d_t = torch.from_numpy(off).cuda(), torch.from_numpy(tails).cuda()
    out = torch.full((1,), 41, dtype=torch.int64, device="cuda")
    stream = torch.cuda.current_stream().cuda_stream
    with waits_give_up(), pytest.raises(xt.XtError) as err:
        xt.count_device(NV, d_off, d_t, out, accumulate=accumulate, stream=stream)
    assert err.value.status == xt.XT_ERR_TIMEOUT
    assert int(out) == 41, "the counter is left alone"
    xt.count_device(NV, d_off, d_t, out, accumulate=accumulate, stream=stream)
    assert int(out) == want + (41 if accumulate else 0)


@pytest.mark.parametrize("form", ["edges", "edges by id", "csr", "canonical csr"])
def test_a_build_leaves_an_asynchronous_timeout_to_the_next_count(dense, form):
    """A count_async whose waits ran out is not an error of the next build's
    input: the build succeeds (and still refuses bad input), the next
    synchronous count reports the timeout, and the one after is exact."""
    import torch
    import xxtric_b200 as xt
    off, tails, (want, _) = dense
    with xt.Context(0) as c:
        g = c.graph_from_csr(off, tails)
        total = torch.zeros(1, dtype=torch.int64, device="cuda")
        torch.cuda.synchronize()
        with waits_give_up():
            g.count_async(total)
        c.synchronize()
        if form.startswith("edges"):
            orient = 0 if form == "edges by id" else 1
            rows = np.array([0, 0, 1], np.int32), np.array([1, 2, 2], np.int32)
            with pytest.raises(xt.XtError) as err:
                c.graph_from_edges(2, *rows, orient)
            assert err.value.status == xt.XT_ERR_INVALID
            small = c.graph_from_edges(3, *rows, orient)
        else:
            o, t = np.array([0, 2, 4, 6]), np.array([1, 2, 0, 2, 0, 1])
            with pytest.raises(xt.XtError) as err:
                c.graph_from_csr(o[[0, 2, 1, 3]], t, canonical=form != "csr")
            assert err.value.status == xt.XT_ERR_INVALID
            small = c.graph_from_csr(o, t, canonical=form != "csr")
        with pytest.raises(xt.XtError) as err:
            small.count()
        assert err.value.status == xt.XT_ERR_TIMEOUT
        assert small.count() == 1 and g.count() == want
        small.free()
        g.free()
