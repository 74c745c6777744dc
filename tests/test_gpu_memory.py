"""Calls on a GPU whose memory others hold (option "hold_back_memory": device
allocations that would leave less than that free fail on the host): what runs
without the spare memory, and that its results are those of a roomy device."""
import numpy as np
import pytest

from falconnpp_b200 import capi, synth

pytestmark = pytest.mark.gpu


def _budget(g, nbytes):
    """Leaves the library nbytes of device memory from here on (None: all)."""
    import torch
    torch.cuda.synchronize()
    g.set_option("hold_back_memory", 0 if nbytes is None else max(1, torch.cuda.mem_get_info()[0] - nbytes))


@pytest.fixture
def handle():
    made = []

    def make(X, *params):
        g = capi.Index(*X.shape)
        g.set_index_param(*params, 8, 42)
        made.append(g)
        return g

    yield make
    for g in made:
        g.set_option("hold_back_memory", 0)
        g.close()


@pytest.mark.parametrize("d", [128, 127])
def test_host_build_needs_no_more_than_a_device_build(handle, d):
    # the copy of the host data must not lie beside the ids and the build's scratch
    import torch
    X = synth.mixture(300_000, d, n_centres=16, seed=0)
    x = torch.from_numpy(X).cuda()
    g = handle(X, 6, 64, 50, 0.05, 1)
    g.build(X)
    want = (g.dump_center(), *g.dump_tables())

    def fits(build, nbytes):
        g.clear()
        _budget(g, nbytes)
        try:
            build()
        except capi.FppError as e:
            assert e.code == -4
            return False
        finally:
            _budget(g, None)
        return True

    lo, hi = 32 << 20, 1 << 30
    assert fits(lambda: g.build_device(x.data_ptr()), hi)
    while hi - lo > 2 << 20:
        mid = (lo + hi) // 2
        lo, hi = (lo, mid) if fits(lambda: g.build_device(x.data_ptr()), mid) else (mid, hi)
    assert fits(lambda: g.build(X), hi + (8 << 20))
    for a, b in zip(want, (g.dump_center(), *g.dump_tables()), strict=True):
        assert np.array_equal(a, b)


def test_index_without_its_optional_arrays(handle, tmp_path):
    # little memory beside the index: no int8 rows and no hash matrix, the same
    # results, whether it was built or loaded so
    X = synth.mixture(30_000, 100, n_centres=16, seed=0)
    Q = synth.mixture(700, 100, n_centres=16, seed=1)
    roomy, tight, loaded = (handle(X, 20, 128, 100, 0.05, 2) for _ in range(3))
    roomy.build(X)
    roomy.save(str(tmp_path / "index"))
    _budget(tight, 300 << 20)
    tight.build(X)
    loaded.load(str(tmp_path / "index"))
    _budget(tight, None)
    assert [roomy.info()[k] for k in ("screen_rows", "hash_matrix")] == [True, True]
    for g in (tight, loaded):
        assert [g.info()[k] for k in ("screen_rows", "hash_matrix")] == [False, False]
        for a, b in zip(roomy.dump_tables(), g.dump_tables(), strict=True):
            assert np.array_equal(a, b)
        for nq in (5, 700):
            for qp in (3, 20):
                for form in ((0, 0, 4), (1, 0, 4), (1, 1, 2), (1, 2, 2)):
                    got = []
                    for h in (roomy, g):
                        h.set_qprobes(qp)
                        h.set_query_form(*form)
                        got.append(h.query(Q[:nq], 10))
                    assert np.array_equal(*got), (nq, qp, form)


def test_plain_query_whose_batched_scratch_does_not_fit(handle):
    # one bucket of nearly all points makes the fused kernel's per-block lists
    # large (they allow for qProbes of the largest), the candidates found are few
    X = synth.mixture(200_000, 32, n_centres=64, seed=0)
    X[:150_000] = X[0] * np.random.default_rng(0).uniform(0.5, 1.5, (150_000, 1)).astype(np.float32)
    Q = synth.mixture(2000, 32, n_centres=64, seed=1)
    Q = Q[Q @ X[0] < 0][:500]
    g = handle(X, 10, 64, 20_000, 0.05, 1)
    g.build(X)
    g.set_qprobes(8)
    want = g.query(Q, 10)
    batched = g.stats(1)
    _budget(g, 8 << 20)
    assert np.array_equal(g.query(Q, 10), want)  # the workspace is there
    g.clear()
    _budget(g, None)
    g.build(X)
    g.set_qprobes(8)
    import torch
    q = torch.from_numpy(Q).cuda()
    out = torch.full((500, 10), -7, dtype=torch.int32, device="cuda")
    _budget(g, 200 << 20)
    got = g.query(Q, 10)
    stats = g.stats(1)
    g.query_device(q.data_ptr(), 500, 10, out.data_ptr())
    _budget(g, None)
    # 8 bytes a candidate for qProbes of the largest bucket, 444 blocks: it cannot have been the fused kernel
    assert 8 * 8 * g.info()["max_kept"] * 444 > 200 << 20
    assert np.array_equal(got, want) and np.array_equal(out.cpu().numpy(), want)
    assert np.array_equal(stats[:4], batched[:4])  # candidates, unique, empty, probes
