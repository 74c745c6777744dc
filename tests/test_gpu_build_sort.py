"""Build: the key selection, the pairs in registers and the bucket sorts, where
they can go wrong, against the oracle bit for bit (hash codes, scores, bucket
contents in the reference's order): every iProbes around the register forms,
n_proj below and at fhtDim, buckets around the warp, shared-memory and repair
sizes, chunks of one table and of several, and more ties than the deferred
repairs hold."""
import numpy as np
import pytest

from falconnpp_b200 import synth
from tests.helpers import build_both, compare_build

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("iprobes", [1, 2, 3, 4])
@pytest.mark.parametrize("d,D", [(20, 32), (48, 64), (100, 64), (128, 128), (200, 256), (300, 64), (600, 16)])
def test_selection(d, D, iprobes):
    X = synth.mixture(1500, d, n_centres=8, seed=0)
    X[100] = 0.0                                  # every coordinate ties
    X[200] = X[201]
    o, g, codes, scores = build_both(X, 3, D, 20, 0.05, iprobes)
    compare_build(o, g, codes, scores)
    g.close()


@pytest.mark.parametrize("n", [31, 33, 64, 65, 513, 900, 2100, 7100, 9000])
def test_bucket_sizes(n):
    # n_proj 1: four buckets per table hold everything
    X = synth.mixture(n, 6, n_centres=3, seed=n)
    o, g, codes, scores = build_both(X, 2, 1, n // 2, 0.3, 1)
    compare_build(o, g, codes, scores)
    g.close()


def test_integer_ties_everywhere():
    X = synth.p0_integer(20000, 8, xmax=2)
    o, g, codes, scores = build_both(X, 4, 8, 300, 0.2, 3)
    compare_build(o, g, codes, scores)
    g.close()
