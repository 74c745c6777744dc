"""Build: buckets beyond a block's shared memory (tiles of 8,192 entries and
their merges), against the oracle bit for bit.  The points are multiples of one
vector of fhtDim coordinates and of its negative, so every table has two
buckets: one entry under, at and over one, two and four tiles, ragged ones, and
two buckets of different sizes; with all scores different and with few values
(every bucket then goes through the heap replay of the largest class)."""
import numpy as np
import pytest

from tests.helpers import build_both, compare_build

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("values", [0, 40])
@pytest.mark.parametrize("pos,neg", [(8191, 8191), (8192, 8192), (8193, 8193), (16_384, 16_385), (24_577, 8193),
                                     (32_769, 32_768), (50_001, 33), (9000, 70_000)])
def test_bucket_of_tiles(pos, neg, values):
    rng = np.random.default_rng(pos + neg)
    v = rng.standard_normal(8).astype(np.float32) + 2.0
    c = rng.uniform(1.0, 2.0, pos + neg) if values == 0 else rng.integers(1, values + 1, pos + neg) / values + 1.0
    # the mean is near zero (the smaller side farther out), so no point changes sides
    c[:pos] *= max(1.0, neg / pos)
    c[pos:] *= -max(1.0, pos / neg)
    X = (rng.permutation(c)[:, None] * v[None, :]).astype(np.float32)
    o, g, codes, scores = build_both(X, 2, 4, 30, 0.3, 1)
    compare_build(o, g, codes, scores)
    assert np.bincount(codes[0].ravel()).max() == max(pos, neg)
    g.close()


def test_several_chunks_and_probes():
    # two huge buckets per table and probe, a chunk of tables at a time
    rng = np.random.default_rng(0)
    X = rng.standard_normal((60_000, 5)).astype(np.float32)
    o, g, codes, scores = build_both(X, 3, 2, 500, 0.2, 2)
    compare_build(o, g, codes, scores)
    for chunk in (1, 2):
        g.set_option("tables_per_chunk", chunk)
        g.set_option("repair_arena", 10_000)
        g.build(X)
        compare_build(o, g, None, None)
    g.close()
