"""Build: the arena and the item lists of the put-off tie repairs run out.
Integer data (ties in nearly every bucket, buckets of one entry to thousands)
with room for a few of them only, so warps compete for the last ranges and the
rest is repaired chunk by chunk: the oracle's tables bit for bit, every time."""
import pytest

from falconnpp_b200 import synth
from tests.helpers import compare_build

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("arena,items", [(1, 0), (600, 0), (5000, 0), (60_000, 0), (0, 1), (0, 40), (3000, 60)])
def test_repairs_beyond_the_room_put_aside(arena, items):
    from falconnpp_b200 import capi
    from oracle import oracle
    X = synth.p0_integer(12_000, 8, xmax=2)
    args = (6, 8, 300, 0.2, 2)
    o = oracle.Index(*X.shape)
    o.set_index_param(*args, 0, 42)
    o.build(X)
    g = capi.Index(*X.shape)
    g.set_index_param(*args, 8, 42)
    g.set_option("repair_arena", arena)
    g.set_option("repair_items", items)
    for chunk in (0, 0, 1, 4):
        g.set_option("tables_per_chunk", chunk)
        g.build(X)
        compare_build(o, g, None, None)
    g.close()
