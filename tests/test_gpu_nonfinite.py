"""Vectors that rotate to NaN, beside ordinary ones in the same warp: queries
with NaN or infinite entries, and finite data whose rotation overflows.  A group
of lanes that finds no comparable coordinate must stay with its warp to the end
of the selection; the ordinary vectors' results are those they get without
such neighbours, and every form answers the others alike."""
import numpy as np
import pytest

from falconnpp_b200 import capi, synth

pytestmark = pytest.mark.gpu


def _index(X, L, D, iprobes):
    g = capi.Index(*X.shape)
    g.set_index_param(L, D, 40, 0.05, iprobes, 8, 42)
    g.build(X)
    return g


def _device(g, Q, k, qp, form, split):
    import torch
    g.set_query_form(*form)
    g.set_option("split_hash", split)
    dq = torch.from_numpy(np.ascontiguousarray(Q)).cuda()
    ids = torch.full((len(Q), k), -7, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    g.query_batched(dq.data_ptr(), len(Q), None, None, k, qp, ids.data_ptr(), k)
    g.set_option("split_hash", 1)
    g.set_query_form(0, 0, 4)
    return ids.cpu().numpy()


# one to five probes per layer
@pytest.mark.parametrize("d,D", [(20, 32), (48, 64), (100, 128), (200, 256), (300, 512)])
def test_queries(d, D):
    L = 6
    X = synth.mixture(3000, d, n_centres=16, seed=0)
    Q = synth.mixture(64, d, n_centres=16, seed=1)
    odd = np.array([0, 1, 3, 9, 17, 33, 34, 35])
    rest = np.setdiff1d(np.arange(64), odd)
    Q[odd, 0] = [np.nan, np.inf, -np.inf, np.nan, np.inf, np.nan, -np.inf, np.nan]
    Q[33] = np.nan
    g = _index(X, L, D, 2)
    for qp in (3, 6, 12, 27, 60):
        g.set_qprobes(qp)
        alone = g.query_dump(Q[rest], 10, qp)["topk"]
        ref = g.query_dump(Q, 10, qp)["topk"]
        assert np.array_equal(ref[rest], alone), qp
        assert np.array_equal(g.query(Q, 10), ref), qp
        for split in (1, 0):
            assert np.array_equal(_device(g, Q, 10, qp, (1, 0, 4), split), ref), (qp, split)
            for precision in (1, 2):
                assert np.array_equal(_device(g, Q, 10, qp, (1, precision, 4), split)[rest],
                                      _device(g, Q[rest], 10, qp, (1, precision, 4), split)), (qp, split, precision)
    g.close()


@pytest.mark.parametrize("iprobes", [1, 2, 3, 4, 6])
@pytest.mark.parametrize("d,D", [(24, 32), (64, 64), (200, 256), (100, 16)])
def test_data_whose_rotation_overflows(d, D, iprobes):
    # pairs of opposite points, so that the centre stays where it was
    from oracle import oracle
    X = synth.mixture(800, d, n_centres=8, seed=0)
    huge = np.arange(100, 740, 80)
    X[huge] *= np.float32(3e37)
    X[huge + 1] = -X[huge]
    rest = np.setdiff1d(np.arange(800), np.concatenate([huge, huge + 1]))
    o = oracle.Index(*X.shape)
    o.set_index_param(3, D, 20, 0.05, iprobes, 0, 42)
    o.build(X)
    g = capi.Index(*X.shape)
    g.set_index_param(3, D, 20, 0.05, iprobes, 8, 42)
    codes, scores = g.build_dump_hash(X)
    co, so = o.hash_codes()
    assert np.array_equal(codes[:, rest], co[:, rest])
    assert np.array_equal(scores[:, rest].view(np.uint32), so[:, rest].view(np.uint32))
    assert codes.min() >= 0 and codes.max() < 4 * D * D
    g.close()
