"""Forms that share kernels, each against a path of its own.

Plain queries, the batched FP32 form and, for up to 222 queries, both through
clusters run the same kernels, so comparing them with one another shows little:
here they are compared with query_dump, the three-kernel path (itself pinned to
the oracle).  The int8 screen of the fused kernel and the verified hash without
the rotation matrices run at batch sizes that reach them, and clusters at row
sizes beside the usual one.  Exact comparison everywhere."""
import numpy as np
import pytest

from falconnpp_b200 import capi, synth
from tests.test_gpu_screen import _check as check_screen
from tests.test_gpu_tc_hash import _check as check_hash
from tests.test_gpu_tc_hash import _rehashed

pytestmark = pytest.mark.gpu


def _index(X, L, D, min_size, alpha, iprobes):
    g = capi.Index(*X.shape)
    g.set_index_param(L, D, min_size, alpha, iprobes, 8, 42)
    g.build(X)
    return g


def _batched(g, Q, k, qp, precision=0, mult=4, graph=0, ks=None, qps=None):
    import torch
    g.set_query_form(1, precision, mult)
    g.set_option("use_graph", graph)
    dev = [None if v is None else torch.from_numpy(np.ascontiguousarray(v)).cuda() for v in (Q, ks, qps)]
    ids = torch.full((len(Q), k), -7, dtype=torch.int32, device="cuda")
    val = torch.zeros((len(Q), k), dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    g.query_batched(dev[0].data_ptr(), len(Q), *[None if v is None else v.data_ptr() for v in dev[1:]], k, qp,
                    ids.data_ptr(), k, val.data_ptr())
    g.set_query_form(0, 0, 4)
    return ids.cpu().numpy(), val.cpu().numpy().view(np.uint32)


def _odd_queries(Q):
    """The first of them zero, tiny, huge and not finite."""
    Q = Q.copy()
    Q[0] = 0.0
    Q[1] *= 1e-30
    Q[2] *= 1e25
    Q[3, 0] = np.inf
    Q[4, 0] = -np.inf
    Q[5, 0] = np.nan
    Q[6] = np.nan
    return Q


@pytest.mark.parametrize("nq", [40, 300, 1000])
@pytest.mark.parametrize("n,d,L,D,min_size,alpha,iprobes", [
    (3000, 24, 4, 32, 20, 0.01, 1),
    (5000, 64, 6, 64, 5, 0.05, 2),
    (4000, 200, 3, 256, 50, 0.01, 3),
    (2000, 100, 5, 128, 10, 0.5, 4),
])
def test_plain_and_fp32_against_three_kernels(n, d, L, D, min_size, alpha, iprobes, nq):
    X = synth.mixture(n, d, n_centres=16, seed=0)
    Q = _odd_queries(synth.mixture(nq, d, n_centres=16, seed=1))
    g = _index(X, L, D, min_size, alpha, iprobes)
    for qp in (1, 5, 3 * L):
        g.set_qprobes(qp)
        ref = g.query_dump(Q, 10, qp)
        assert np.array_equal(g.query(Q, 10), ref["topk"]), qp
        for graph in (0, 1):
            ids, val = _batched(g, Q, 10, qp, graph=graph)
            assert np.array_equal(ids, ref["topk"]), (qp, graph)
            assert np.array_equal(val[7:], ref["topk_val"].view(np.uint32)[7:]), (qp, graph)
    g.close()


@pytest.mark.parametrize("nq", [60, 260])
def test_ties_against_three_kernels(nq):
    X = synth.p0_integer(2000, 32, xmax=7)
    Q = synth.p0_queries(nq, 32, qmax=3)
    g = _index(X, 5, 32, 10, 0.02, 3)
    for qp in (2, 7, 40):
        g.set_qprobes(qp)
        ref = g.query_dump(Q, 20, qp)
        assert np.array_equal(g.query(Q, 20), ref["topk"])
        ids, val = _batched(g, Q, 20, qp)
        assert np.array_equal(ids, ref["topk"])
        assert np.array_equal(val, ref["topk_val"].view(np.uint32))
    g.close()


def test_mixed_batch_against_three_kernels():
    X = synth.mixture(20000, 100, n_centres=32, seed=0)
    Q = synth.mixture(700, 100, n_centres=32, seed=1)
    g = _index(X, 10, 128, 30, 0.01, 3)
    rng = np.random.default_rng(3)
    ks = rng.choice([1, 10, 100], size=len(Q)).astype(np.int32)
    qps = rng.choice([5, 10, 20, 80], size=len(Q)).astype(np.int32)
    ids, _ = _batched(g, Q, 100, 80, ks=ks, qps=qps)
    for kk in (1, 10, 100):
        for qq in (5, 10, 20, 80):
            sel = np.where((ks == kk) & (qps == qq))[0]
            g.set_qprobes(qq)
            assert np.array_equal(ids[sel, :kk], g.query_dump(Q[sel], kk, qq)["topk"]), (kk, qq)
    g.close()


@pytest.mark.parametrize("d", [20, 33, 216, 217, 248, 249, 505, 512])
def test_screen_of_the_fused_kernel_row_sizes(d):
    X = synth.mixture(20000, d, n_centres=16, seed=0)
    Q = synth.mixture(230, d, n_centres=16, seed=1)
    check_screen(X, Q, 10, 64, 10, 12)


@pytest.mark.parametrize("k", [1, 150, 600, 1024])
def test_screen_of_the_fused_kernel_k(k):
    X = synth.mixture(30000, 96, n_centres=8, seed=0)
    Q = synth.mixture(230, 96, n_centres=8, seed=1)
    check_screen(X, Q, 10, 64, k, 30, min_size=200)


def test_data_that_defeats_the_screen_of_the_fused_kernel():
    check_screen(synth.p0_integer(6000, 32, xmax=3), synth.p0_queries(240, 32, qmax=2), 8, 32, 10, 40)
    Q = synth.mixture(240, 100, n_centres=8, seed=1)
    X = synth.mixture(20000, 100, n_centres=8, seed=0)
    X[1::2] = X[::2]
    check_screen(X, Q, 10, 64, 10, 20)
    X = synth.mixture(20000, 100, n_centres=8, seed=0)
    X[::501] *= 1e6
    X[7] *= 1e15
    Q[:8] = 0.0
    Q[:7, :7] = np.eye(7)
    Q[8] *= 1e20
    Q[9] *= 1e-25
    Q[10] *= 1e-40
    check_screen(X, Q, 10, 64, 10, 20)


@pytest.mark.parametrize("precision", [0, 1, 2])
@pytest.mark.parametrize("d", [20, 100, 217, 256, 512])
def test_clusters_row_sizes(d, precision):
    # 1, 18, 37 and 222 queries: clusters of 8, 8, 4 and 2 blocks; 600: none
    X = synth.mixture(20000, d, n_centres=16, seed=0)
    Q = synth.mixture(600, d, n_centres=16, seed=1)
    g = _index(X, 12, 64, 200, 0.05, 2)
    for k, qp in ((1, 1), (20, 6), (50, 100)):
        ids, val = _batched(g, Q, k, qp, precision, 2)
        for nq in (1, 18, 37, 222):
            few = _batched(g, Q[:nq], k, qp, precision, 2)
            assert np.array_equal(few[0], ids[:nq]), (k, qp, nq)
            assert np.array_equal(few[1], val[:nq]), (k, qp, nq)
    g.close()


@pytest.mark.parametrize("L,D", [(8, 64), (31, 32), (65, 64), (128, 64)])
def test_verified_hash_without_matrices(L, D):
    # fhtDim 256 with fewer than 128 projections: no matrices, so the rotation
    # per query, from 257 queries on
    X = synth.mixture(20_000, 200, n_centres=64, seed=2)
    Q = synth.mixture(300, 200, n_centres=64, seed=3)
    Q[:8] *= np.array([0.0, 1e-25, 1e-16, 1e-6, 1.0, 1e6, 1e16, 1e25], np.float32)[:, None]
    g = _index(X, L, D, 50, 0.01, 3)
    assert not g.info()["hash_matrix"]
    for qp in (1, 3, L // 2):
        check_hash(g, Q, 10, qp, precisions=(0, 2))
    assert len(Q) <= _rehashed(g, Q, 10, 1) <= len(Q) * L
    g.close()


def test_verified_hash_without_matrices_ties():
    X = synth.p0_integer(4000, 200, xmax=15)
    Q = synth.p0_queries(300, 200, qmax=3)
    Q[0] = 0
    g = _index(X, 8, 64, 20, 0.02, 3)
    for qp in (1, 2, 3, 4):
        check_hash(g, Q, 20, qp)
    assert _rehashed(g, Q, 20, 2) >= 2 * len(Q)
    g.close()


@pytest.mark.parametrize("d,D", [(100, 128), (200, 256), (250, 512)])
def test_hash_matrix_of_a_loaded_index(tmp_path, d, D):
    X = synth.mixture(6000, d, n_centres=32, seed=4)
    Q = synth.mixture(400, d, n_centres=32, seed=5)
    built = _index(X, 20, D, 40, 0.02, 2)
    built.save(str(tmp_path / "index"))
    g = capi.Index(*X.shape)
    g.load(str(tmp_path / "index"))
    assert g.info()["hash_matrix"]
    for qp in (1, 5, 10):
        check_hash(g, Q, 10, qp)
    assert _rehashed(g, Q, 10, 1) >= len(Q)
    for h in (built, g):
        h.close()
