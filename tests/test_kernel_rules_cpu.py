"""Sizes and choices that the kernels library settles on the host, before any launch: they need no device."""
import pytest

from hartsyinference_b200.ops import _native as N

pytestmark = pytest.mark.skipif(not N.available(), reason="kernels library not built")


@pytest.mark.parametrize("heads", [16, 32, 64, 128])
@pytest.mark.parametrize("rows", [1, 8, 16, 32, 48, 96, 128, 200])
def test_latent_attention_ranges_do_not_grow_with_the_longest_length(rows, heads):
    """A step made for 32768 keys runs with a few hundred as well: blocks for all of them at a time, two on a processor, not more; and rows
    of unequal lengths are cut as long as that leaves processors idle."""
    blocks = rows * max(1, heads // 32)
    for most in (2304, 8192, 32768):
        s = N.lib().b200_mla_pick_splits(rows, heads, most)
        assert 1 <= s <= max(1, -(-2 * 148 // blocks))
        assert s * blocks >= min(2 * 148, 32 * blocks)
