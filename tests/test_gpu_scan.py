"""The threshold scan behind the brute-force top-k (low precision and FP64).

Integer data whose BF16 / FP32 scores are exact pin the kept set and its order
(score desc, id asc) against a stable FP64 sort, with equal scores everywhere,
at row and query counts around the tiles and for every sampling stride; data
that the scan cannot settle (zero queries, thousands of equal scores, huge
norms) must give the same results through the per-point kernels."""
import numpy as np
import pytest

from falconnpp_b200 import capi, synth

pytestmark = pytest.mark.gpu


def _exact(X, Q, k):
    """Top k by (score desc, id asc) in FP64."""
    s = X.astype(np.float64) @ Q.astype(np.float64).T
    ids = np.argsort(-s, axis=0, kind="stable")[:k].T
    return ids.astype(np.int32), np.take_along_axis(s.T, ids, axis=1)


def _truth(X, Q, k):
    import torch
    x, q = torch.from_numpy(X).cuda(), torch.from_numpy(Q).cuda()
    ids = torch.full((len(Q), k), -7, dtype=torch.int32, device="cuda")
    val = torch.zeros((len(Q), k), dtype=torch.float64, device="cuda")
    capi.bruteforce_topk_f64(x.data_ptr(), len(X), X.shape[1], q.data_ptr(), len(Q), k, ids.data_ptr(), val.data_ptr())
    return ids.cpu().numpy(), val.cpu().numpy()


@pytest.mark.parametrize("n,d,nq,k", [(300_001, 16, 130, 20), (100_000, 48, 128, 20), (40_000, 33, 257, 5),
                                      (20_100, 256, 1, 1), (9_000, 100, 300, 20), (60_000, 7, 64, 100)])
def test_truth(n, d, nq, k):
    rng = np.random.default_rng(n)
    X = rng.standard_normal((n, d)).astype(np.float32)
    Q = rng.standard_normal((nq, d)).astype(np.float32)
    ids, val = _truth(X, Q, k)
    ref, rv = _exact(X, Q, k)
    assert np.array_equal(ids, ref)
    # d products and sums in another order: d 2^-52 of the sum of magnitudes
    assert np.all(np.abs(val - rv) <= d * 2.0 ** -52 * np.abs(Q).sum(1)[:, None] * np.abs(X).max())


def test_truth_that_the_scan_cannot_settle():
    rng = np.random.default_rng(0)
    X = rng.integers(-3, 4, (50_000, 24)).astype(np.float32)
    X[1000:30_000] = X[999]                      # thousands of equal scores
    Q = rng.integers(-3, 4, (40, 24)).astype(np.float32)
    Q[3] = 0.0
    Q[4] = X[999]
    ids, val = _truth(X, Q, 20)
    ref, rv = _exact(X, Q, 20)
    assert np.array_equal(ids, ref) and np.array_equal(val, rv)
    X[7] *= 1e20                                 # out of the scan's range
    Q[5] *= 1e-20
    ids, val = _truth(X, Q, 20)
    ref, rv = _exact(X, Q, 20)
    assert np.array_equal(ids, ref)


@pytest.mark.parametrize("precision", [1, 2])
@pytest.mark.parametrize("n,d,nq,k,mult", [(200_001, 20, 200, 20, 4), (70_000, 32, 129, 10, 4), (12_000, 64, 64, 10, 2)])
def test_lowp_exact_integers(precision, n, d, nq, k, mult):
    import torch
    # E4M3 holds -3..3 times the row scale 3 / 448 exactly enough to order
    # integer scores only in BF16; FP8 is checked on sign data (+-1)
    rng = np.random.default_rng(d)
    half = rng.integers(-3, 4, (n // 2, d)) if precision == 1 else rng.choice([-1, 1], (n // 2, d))
    X = np.empty((n // 2 * 2, d), np.float32)
    X[0::2], X[1::2] = half, -half               # sign symmetric: the centre is exactly 0
    Q = (rng.integers(-3, 4, (nq, d)) if precision == 1 else rng.choice([-1, 1], (nq, d))).astype(np.float32)
    Q[0] = 0.0
    g = capi.Index(*X.shape)
    g.set_index_param(1, 16, 10, 0.1, 1, 8, 1)
    g.build(X)
    dq = torch.from_numpy(Q).cuda()
    ids = torch.full((nq, k), -7, dtype=torch.int32, device="cuda")
    val = torch.zeros((nq, k), dtype=torch.float32, device="cuda")
    g.bruteforce_lowp(dq.data_ptr(), nq, k, precision, mult, ids.data_ptr(), val.data_ptr())
    g.close()
    ref, rv = _exact(X, Q, k)
    assert np.array_equal(val.cpu().numpy().astype(np.float64), rv)
    assert np.array_equal(ids.cpu().numpy(), ref)
