"""Sizes and choices that the kernels library settles on the host, before any launch: they need no device."""
import pytest

from hartsyinference_b200 import config
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


def test_prompt_layers_refuse_scratch_of_another_reduce_form():
    """The ranges that products leave unsummed need scratch only in one reduce form, which can be switched between the call that asks for
    the size and the launch: the launch then returns an error before it touches anything."""
    L, sizes, ws = N.lib(), (896, 14, 2, 64, 4864), 64 << 20
    try:
        L.b200_gemm_set_external_reduce(0)
        small = L.b200_dense_layers_scratch(29, *sizes, ws)
        L.b200_gemm_set_external_reduce(1)
        need = L.b200_dense_layers_scratch(29, *sizes, ws)
        assert small < need
        hidden, hq, hkv, d, ffn = sizes
        args = (None, None, None, None, None, 0, 0, None, None, None, None, None, None, 29, 1, 29, 29, 24, hidden, hq, hkv, d, ffn, d, 0, 16, 4, 64, 0, 0,
                1e-6, 1e4, 0.125, None, ws, None)
        assert L.b200_dense_layers(*args, small, None, None) == -14
    finally:
        L.b200_gemm_set_external_reduce(1 if config.get("splitk_second_kernel") else 0)


@pytest.mark.parametrize("hidden,hq,hkv,d,ffn", [(4096, 32, 8, 128, 14336), (8192, 64, 8, 128, 28672), (896, 14, 2, 64, 4864)])
@pytest.mark.parametrize("tokens", [2048, 8192])
def test_prompt_layers_scratch_holds_what_lives_at_once(tokens, hidden, hq, hkv, d, ffn):
    """Long prompts, whose gated product forms the activation itself: four rows of the stream's width, and the larger of what the two halves
    of a layer hold (the packed projection and q, the activation); no gate and up rows."""
    got = N.lib().b200_dense_layers_scratch(tokens, hidden, hq, hkv, d, ffn, 64 << 20)
    assert got <= 2 * tokens * (4 * hidden + max((2 * hq + 2 * hkv) * d, ffn)) + 16 * 256


# both forms measured without filters and with all of them: a cluster where it is a fifth faster with all and at most an eighth slower without
@pytest.mark.parametrize("rows,vocab,cluster", [
    (1, 1000, 0), (8, 2048, 0), (16, 4096, 0), (37, 8192, 0), (48, 16384, 0), (148, 128256, 0), (200, 50257, 0), (200, 202048, 0), (256, 151936, 0), (512, 100352, 0),
    (1, 8192, 1), (8, 16384, 1), (64, 32000, 1), (96, 50257, 1), (64, 128256, 1), (128, 128256, 1), (128, 151936, 1), (1, 256000, 1), (1, 262145, 0), (1 << 28, 32000, 0)])
def test_sampler_form(rows, vocab, cluster):
    assert N.lib().b200_sample_form(rows, vocab) == cluster


# both kernels measured: CTA pairs where they are faster (dtype 0 bf16, 2 fp8)
@pytest.mark.parametrize("m,n,k,dtype,pairs", [
    (300, 4096, 14336, 0, 0), (300, 4096, 8192, 0, 0), (300, 2048, 4096, 0, 0), (129, 4096, 4096, 0, 0), (512, 4096, 18432, 0, 0), (2600, 7168, 14336, 0, 0),
    (640, 28672, 8192, 0, 0), (300, 2048, 8192, 2, 0), (129, 4096, 12288, 2, 0), (300, 6144, 1024, 2, 0), (300, 6144, 256, 2, 0), (128, 28672, 4096, 0, 0),
    (300, 4096, 6144, 0, 1), (300, 3072, 4096, 0, 1), (1024, 1024, 3072, 0, 1), (256, 9216, 3072, 0, 1), (640, 28672, 1024, 0, 1), (2600, 28672, 4096, 0, 1),
    (1024, 1024, 8192, 2, 1), (300, 6144, 2048, 2, 1), (600, 4096, 3072, 2, 1), (4096, 9216, 3072, 2, 1)])
def test_products_on_pairs(m, n, k, dtype, pairs):
    assert N.lib().b200_gemm_on_pairs(m, n, k, dtype) == pairs


@pytest.mark.parametrize("m,n,pays", [(200, 21504, 0), (512, 12288, 0), (1024, 13824, 0), (1651, 3072, 0), (1651, 6144, 1), (2560, 3072, 1), (4608, 12288, 1), (14040, 13824, 1)])
def test_quantising_epilogue_pays(m, n, pays):
    assert N.lib().b200_gemm_quant_pays(m, n) == pays
