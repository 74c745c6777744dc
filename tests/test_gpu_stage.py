"""Host data of 64 MB and more reaches the device through staged pinned
buffers from a handle's second build on (128 MB: from the first): pieces that
do not divide the size, another build on the same buffers, pinned input (not staged), and data under the line must all give the
tables of the build from device memory."""
import numpy as np
import pytest

from falconnpp_b200 import capi

pytestmark = pytest.mark.gpu


def _tables(n, d, build):
    g = capi.Index(n, d)
    g.set_index_param(2, 64, 20, 0.05, 1, 8, 42)
    out = []
    for b in build:
        b(g)
        out.append(g.dump_tables())
    g.close()
    return out


@pytest.mark.parametrize("n,d", [(65537, 256), (83001, 203), (65535, 256), (131075, 257)])
def test_staged_build(n, d):
    import torch
    gen = torch.Generator(device="cuda").manual_seed(n)
    x = torch.randn((n, d), generator=gen, device="cuda")
    y = torch.randn((n, d), generator=gen, device="cuda")
    torch.cuda.synchronize()
    want = _tables(n, d, [lambda g: g.build_device(x.data_ptr()), lambda g: g.build_device(y.data_ptr())])
    pinned = x.cpu().pin_memory()
    hx, hy = x.cpu().numpy(), y.cpu().numpy()
    got = _tables(n, d, [lambda g: g.build(hx), lambda g: g.build(hy), lambda g: g.build(hx),
                         lambda g: g.build(pinned.numpy())])
    for w, h in zip([*want, want[0], want[0]], got, strict=True):
        assert np.array_equal(w[0], h[0]) and np.array_equal(w[1], h[1])
