"""The batched form's workspace over calls of changing shape on one handle:
a replayed graph after calls outside it have moved the buffers inside the
per-batch allocation (its base address may stay the same), against the first
call's results."""
import numpy as np
import pytest

from falconnpp_b200 import capi, synth

pytestmark = pytest.mark.gpu


def _index(L=12, D=64, qp=6):
    X = synth.mixture(20000, 64, n_centres=16, seed=0)
    g = capi.Index(*X.shape)
    g.set_index_param(L, D, 100, 0.05, 2, 8, 42)
    g.build(X)
    g.set_qprobes(qp)
    return g


def _batched(g, dq, nq, k, qp, ids):
    ids.fill_(-7)
    import torch
    torch.cuda.synchronize()
    g.query_batched(dq.data_ptr(), nq, None, None, k, qp, ids.data_ptr(), k)
    return ids.cpu().numpy().copy()


@pytest.mark.parametrize("form,nq,qp", [(0, 601, 6), (0, 640, 6), (0, 700, 6), (0, 880, 6), (1, 222, 20), (1, 200, 26)])
def test_graph_after_calls_that_move_buffers_within_the_allocation(form, nq, qp):
    # 600 queries: less than two waves, so the graph's node has no order array;
    # the call between (a plain query, or a small batch on clusters, which takes
    # no graph) needs a few per cent more of the per-batch buffers
    import torch
    Q = synth.mixture(900, 64, n_centres=16, seed=1)
    dq = torch.from_numpy(Q).cuda()
    ids = torch.zeros((600, 10), dtype=torch.int32, device="cuda")
    small = torch.zeros((nq, 10), dtype=torch.int32, device="cuda")
    g = _index()
    g.query_dump(Q, 10, 6)  # the query buffers of host calls are in place
    g.set_option("use_graph", 1)
    g.set_query_form(1, 2, 4)
    first = _batched(g, dq, 600, 10, 6, ids)
    for _ in range(3):
        if form == 0:
            g.set_query_form(0, 0, 4)
            g.set_qprobes(qp)
            g.query(Q[:nq], 10)
            g.set_qprobes(6)
            g.set_query_form(1, 2, 4)
        else:
            _batched(g, dq, nq, 10, qp, small)
        assert np.array_equal(_batched(g, dq, 600, 10, 6, ids), first)
    g.close()


def test_calls_of_changing_shape_settle_on_one_allocation():
    # few queries with many candidates and long lists, many with few, big lists,
    # mixed batches, plain and batched, in turn: after one round of all of them
    # nothing is allocated any more (an allocation would fail here), and every
    # result stays the first round's
    import torch
    Q = synth.mixture(2000, 64, n_centres=16, seed=1)
    dq = torch.from_numpy(Q).cuda()
    qps = torch.from_numpy(np.random.default_rng(0).integers(1, 41, 2000).astype(np.int32)).cuda()
    ids = torch.zeros((2000, 10), dtype=torch.int32, device="cuda")
    g = _index()

    def device(nq, qp, mixed=False, graph=0):
        g.set_query_form(1, 2, 4)
        g.set_option("use_graph", graph)
        ids.fill_(-7)
        torch.cuda.synchronize()
        g.query_batched(dq.data_ptr(), nq, None, qps.data_ptr() if mixed else None, 10, qp, ids.data_ptr(), 10)
        return ids.cpu().numpy().copy()

    def plain(nq, qp):
        g.set_query_form(0, 0, 4)
        g.set_qprobes(qp)
        return g.query(Q[:nq], 10)

    calls = [lambda: device(1, 60), lambda: device(2000, 2), lambda: device(900, 40, mixed=True),
             lambda: device(30, 1500), lambda: plain(1, 1100), lambda: plain(2000, 3),
             lambda: device(1000, 6, graph=1), lambda: device(223, 25), lambda: plain(300, 6)]
    first = [c() for c in calls]
    try:
        for order in (range(len(calls)), reversed(range(len(calls)))):
            for i in order:
                g.set_option("inject_alloc_failure", 1)
                assert np.array_equal(calls[i](), first[i]), i
    finally:
        g.set_option("inject_alloc_failure", 0)
    g.close()


@pytest.mark.parametrize("D,nq,host,launches", [
    (64, 200, False, 3),     # exact hash, probe cut, clusters
    (64, 600, False, 3),     # exact hash, probe cut, fused kernel
    (64, 1000, False, 5),    # and the order's two kernels
    (128, 1000, False, 7),   # the product hash: rows, product, check
    (128, 5000, True, 16),   # four chunks of it
    (64, 5000, True, 8),     # four chunks of the exact hash
])
def test_launches_are_counted(D, nq, host, launches):
    import torch
    Q = synth.mixture(nq, 64, n_centres=16, seed=1)
    g = _index(D=D)
    g.set_query_form(1, 2, 4)
    if host:
        g.query(Q, 10)
    else:
        dq = torch.from_numpy(Q).cuda()
        ids = torch.zeros((nq, 10), dtype=torch.int32, device="cuda")
        _batched(g, dq, nq, 10, 6, ids)
    assert int(g.stats(1)[6]) == launches
    g.close()
