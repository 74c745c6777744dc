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
