"""Sizes and checks that the kernels library settles on the host, before any launch: they need no device."""
import pytest

from hartsyinference_b200.ops import _native as N

pytestmark = pytest.mark.skipif(not N.available(), reason="kernels library not built")


@pytest.fixture
def ring_of_three():
    from hartsyinference_b200 import config
    N.lib().b200_attn_set_decode_stages(3)
    yield
    N.lib().b200_attn_set_decode_stages(int(config.get("decode_attn_stages")))


def test_even_shares_refuse_a_workspace_of_another_ring_depth(ring_of_three):
    """A ring of two tiles runs half as many blocks again as one of three, each with rows of the workspace: bytes asked for before the
    depth is switched are refused, not written past."""
    L = N.lib()
    sizes = (64, 64, 8, 128, 8192)
    held = L.b200_attn_decode_even_bytes(*sizes)
    L.b200_attn_set_decode_stages(2)
    assert 0 < held < L.b200_attn_decode_even_bytes(*sizes)
    at = 1 << 20                                   # never read: the call ends at its checks
    rc = L.b200_attn_decode_even(at, at, at, at, at, at, 64, 64, 8, 128, 16, 512, at, held, 0.1, 0.0, 0, None, None, 0, None)
    assert rc == -5
