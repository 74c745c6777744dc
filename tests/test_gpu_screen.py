"""The int8 screen of the batched FP32 form: every result must equal the plain
path's bit for bit (ids and FP32 scores), at row sizes around the 16-byte
chunks and the staging limits, with k around the direct-scoring limit, and on
data that defeats the screen (ties, duplicates, outlier norms, one-hot, zero
and huge queries), where the kernel scores every candidate in FP32."""
import numpy as np
import pytest

from falconnpp_b200 import capi, synth

pytestmark = pytest.mark.gpu


def _check(X, Q, L, D, k, qprobes, iprobes=2, min_size=60):
    import torch
    g = capi.Index(*X.shape)
    g.set_index_param(L, D, min_size, 0.05, iprobes, 8, 42)
    g.build(X)
    g.set_qprobes(qprobes)
    ref = g.query_dump(Q, k, qprobes)
    g.set_query_form(1, 0, 4)
    dq = torch.from_numpy(np.ascontiguousarray(Q)).cuda()
    ids = torch.full((len(Q), k), -7, dtype=torch.int32, device="cuda")
    val = torch.zeros((len(Q), k), dtype=torch.float32, device="cuda")
    g.query_batched(dq.data_ptr(), len(Q), None, None, k, qprobes, ids.data_ptr(), k, val.data_ptr())
    g.close()
    assert np.array_equal(ids.cpu().numpy(), ref["topk"])
    assert np.array_equal(val.cpu().numpy().view(np.uint32), ref["topk_val"].view(np.uint32))


@pytest.mark.parametrize("d", [20, 33, 100, 200, 216, 217, 248, 249, 505, 512])
def test_row_sizes(d):
    X = synth.mixture(20000, d, n_centres=16, seed=0)
    Q = synth.mixture(70, d, n_centres=16, seed=1)
    _check(X, Q, 10, 64, 10, 12)


@pytest.mark.parametrize("k", [1, 20, 150, 600, 1024])
def test_k(k):
    X = synth.mixture(30000, 96, n_centres=8, seed=0)
    Q = synth.mixture(40, 96, n_centres=8, seed=1)
    _check(X, Q, 10, 64, k, 30, min_size=200)


def test_isotropic_data_and_big_lists():
    rng = np.random.default_rng(3)
    X = rng.standard_normal((20000, 64)).astype(np.float32)
    Q = rng.standard_normal((40, 64)).astype(np.float32)
    _check(X, Q, 12, 64, 20, 40)
    _check(X, Q, 12, 64, 20, 1500)


@pytest.mark.parametrize("precision", [0, 1, 2])
@pytest.mark.parametrize("nq", [1, 18, 19, 37, 38, 222, 223])
def test_small_batches(nq, precision):
    """Clusters of 8, 4, 2 blocks per query and none: the results of the same
    queries inside a large batch."""
    import torch
    X = synth.mixture(30000, 200, n_centres=16, seed=0)
    Q = synth.mixture(600, 200, n_centres=16, seed=1)
    g = capi.Index(*X.shape)
    g.set_index_param(12, 64, 400, 0.05, 2, 8, 42)
    g.build(X)
    g.set_query_form(1, precision, 2)
    dq = torch.from_numpy(Q).cuda()
    # qProbes 1: few candidates; 6; 300: more unique ids than a set's chains take
    for k, qp in ((1, 1), (20, 6), (50, 300)):
        got, val = [], []
        for n in (600, nq):
            ids = torch.full((n, k), -7, dtype=torch.int32, device="cuda")
            v = torch.zeros((n, k), dtype=torch.float32, device="cuda")
            g.query_batched(dq.data_ptr(), n, None, None, k, qp, ids.data_ptr(), k, v.data_ptr())
            got.append(ids.cpu().numpy()[:nq])
            val.append(v.cpu().numpy()[:nq])
        assert np.array_equal(got[0], got[1]), (k, qp)
        assert np.array_equal(val[0].view(np.uint32), val[1].view(np.uint32)), (k, qp)
    if precision == 0:
        g.set_qprobes(6)
        assert np.array_equal(g.query_dump(Q[:nq], 20, 6)["topk"], got_plain(g, Q[:nq]))
    g.close()


def got_plain(g, Q):
    g.set_query_form(0, 0, 4)
    return g.query(Q, 20)


def test_data_that_defeats_the_screen():
    X = synth.p0_integer(6000, 32, xmax=3)
    _check(X, synth.p0_queries(40, 32, qmax=2), 8, 32, 10, 40)
    X = synth.mixture(20000, 100, n_centres=8, seed=0)
    Q = synth.mixture(48, 100, n_centres=8, seed=1)
    X[1::2] = X[::2]                       # every point twice: ties at every place
    _check(X, Q, 10, 64, 10, 20)
    X = synth.mixture(20000, 100, n_centres=8, seed=0)
    X[::501] *= 1e6                        # a few huge norms: coarse bins for the others
    X[7] *= 1e15
    Q[:8] = 0.0
    Q[:7, :7] = np.eye(7)                  # one-hot queries and a zero query
    Q[8] *= 1e20
    Q[9] *= 1e-25
    Q[10] *= 1e-40
    _check(X, Q, 10, 64, 10, 20)
    _check(X * np.float32(1e-20), Q[11:], 10, 64, 10, 20)
