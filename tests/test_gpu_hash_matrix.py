"""The verified hash from the rotations as matrices (hash_lists_verified).

One FP16 product gives every table's score within a bound; the tables that can
reach the probe cut are hashed in FP32, so the probes, their order, the counts
and the ids are those of the exact hash (option "tc_hash" 0;
src/FalconnPP.cpp:358-582).  Exact comparison, no tolerance.  Sizes: every
fhtDim, features that fill and do not fill the rows (multiples of 8) and the
pipeline's boxes (64 elements), n_proj below and at fhtDim, one query tile and
a ragged second one, table counts of every 32-bit mask word, ties at the cut,
and queries of no, tiny, huge and non-finite norm.
"""
import numpy as np
import pytest

from falconnpp_b200 import capi, synth

pytestmark = pytest.mark.gpu


def _run(g, Q, k, qp, tc):
    import torch
    g.set_option("tc_hash", tc)
    g.set_qprobes(qp)
    nq = len(Q)
    dq = torch.from_numpy(np.ascontiguousarray(Q)).cuda()
    out = torch.full((nq, k), -9, dtype=torch.int32, device="cuda")
    probes = torch.zeros((nq, qp), dtype=torch.int32, device="cuda")
    counts = torch.zeros((nq, 2), dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    g.query_batched_dump(dq.data_ptr(), nq, k, out.data_ptr(), None, probes.data_ptr(), counts.data_ptr(), 0)
    torch.cuda.synchronize()
    return out.cpu().numpy(), probes.cpu().numpy(), counts.cpu().numpy()


def _same(g, Q, qps, k=10):
    g.set_query_form(1, 2, 4)
    for qp in qps:
        for a, b, what in zip(_run(g, Q, k, qp, 1), _run(g, Q, k, qp, 0), ("ids", "probes", "counts")):
            bad = np.where((a != b).any(1))[0]
            assert len(bad) == 0, (what, qp, bad[:5])


def _index(X, L, D):
    g = capi.Index(*X.shape)
    g.set_index_param(L, D, 40, 0.02, 2, 8, 42)
    g.build(X)
    return g


@pytest.mark.parametrize("d,D,L,nq", [(1, 128, 4, 300), (9, 128, 31, 257), (64, 128, 32, 511), (127, 128, 33, 513),
                                      (128, 128, 128, 700), (129, 256, 65, 300), (200, 128, 100, 300),
                                      (200, 256, 100, 1025), (255, 256, 127, 300), (256, 256, 96, 300),
                                      (100, 512, 40, 300), (250, 512, 128, 400), (200, 256, 2, 300)])
def test_probes_equal_exact_hash(d, D, L, nq):
    X = synth.mixture(6000, d, n_centres=32, seed=4)
    Q = synth.mixture(nq, d, n_centres=32, seed=5)
    Q[0] = 0.0
    Q[1] *= 1e-30
    Q[2] *= 1e25
    Q[3] *= 1e-18
    Q[4, 0] = np.inf
    Q[5, 0] = np.nan
    Q[6] = X[0]
    g = _index(X, L, D)
    _same(g, Q, sorted({1, min(3, L // 2), L // 2}))
    g.set_option("stage_timing", 1)
    _run(g, Q, 10, 1, 1)
    # the path is the one under test: it hashed tables again, the probed ones
    # of every query at least
    assert nq <= int(g.stats(1)[10]) <= nq * L
    g.close()


@pytest.mark.parametrize("d,D", [(100, 128), (200, 256), (200, 512)])
def test_ties_equal_exact_hash(d, D):
    # small integers: coordinates and scores tie, at the cut too
    X = synth.p0_integer(3000, d, xmax=9)
    Q = synth.p0_queries(300, d, qmax=2)
    Q[0] = 0
    Q[1] = 0
    Q[1, 0] = 1
    g = _index(X, 16, D)
    _same(g, Q, (1, 2, 5, 8))
    g.close()


def test_many_queries_in_parts():
    # more queries than the scratch of the product holds at a time
    X = synth.mixture(3000, 24, n_centres=16, seed=6)
    Q = synth.mixture(33_001, 24, n_centres=16, seed=7)
    g = _index(X, 6, 128)
    _same(g, Q, (1, 3))
    g.close()
