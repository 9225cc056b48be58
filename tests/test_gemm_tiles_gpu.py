"""Large-token products at the edges of their tiles, bands and strips, against the fp32 statement."""
import pytest
import torch

from hartsyinference_b200 import ops
from hartsyinference_b200.ops import reference as R

pytestmark = pytest.mark.gpu


# (tokens, features): the 128 x 256 tile starts at one tile per SM; 2048 tokens are one band; features that are no
# multiple of 32 or 8 leave chunks to the elementwise store
@pytest.mark.parametrize("m,n", [(2049, 2432), (2050, 2328), (4097, 1184), (129, 136), (2177, 2180), (300, 20000)])
@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("act,act_from", [(None, 0), ("gelu_tanh", 0), ("gelu_tanh", 128), ("silu", 12), ("tanh", 64)])
def test_epilogue_and_tiles(m, n, fp8, act, act_from):
    torch.manual_seed(m)
    k = 256
    x = torch.randn(m, k, device="cuda").to(torch.bfloat16)
    w = ops.LinearWeight.from_dense((torch.randn(n, k, device="cuda") * k ** -0.5).to(torch.bfloat16),
                                    torch.randn(n, device="cuda").to(torch.bfloat16), fp8=fp8)
    gate = torch.randn(n, device="cuda").to(torch.bfloat16)
    res = torch.randn(m, n, device="cuda").to(torch.bfloat16)
    xq = ops.quant_fp8_act(x) if fp8 else x
    y = ops.linear(xq, w, act=act, act_from=act_from, gate=gate, residual=res).float()
    ref = R.linear(xq.data if fp8 else x, w.weight, w.scale, xq.scales_fp32() if fp8 else None, w.bias, act, gate, res, torch.float32,
                   act_from=act_from)
    assert torch.allclose(y, ref, rtol=2 ** -7, atol=2 ** -7), (y - ref).abs().max()      # one rounding to bf16; fp32 sums of 256


# tiles of CTA pairs: the fewest that go there, one K block, a K tail, rows and features that end inside a tile, both
# accumulators in turn
@pytest.mark.parametrize("m,n,k", [(256, 4096, 64), (257, 4104, 192), (385, 9232, 136), (2100, 1984, 4096), (5000, 3856, 328), (9473, 2304, 1024)])
@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("full", [False, True])
def test_pair_tiles(m, n, k, fp8, full):
    torch.manual_seed(m)
    k = -(-k // 128) * 128 if fp8 else k
    n = n if not fp8 else -(-n // 16) * 16
    x = torch.randn(m, k, device="cuda").to(torch.bfloat16)
    vec = lambda: torch.randn(n, device="cuda").to(torch.bfloat16) if full else None
    w = ops.LinearWeight.from_dense((torch.randn(n, k, device="cuda") * k ** -0.5).to(torch.bfloat16), vec(), fp8=fp8)
    gate, act = vec(), "gelu_tanh" if full else None
    res = torch.randn(m, n, device="cuda").to(torch.bfloat16) if full else None
    xq = ops.quant_fp8_act(x) if fp8 else x
    y = ops.linear(xq, w, act=act, gate=gate, residual=res).float()
    ref = R.linear(xq.data if fp8 else x, w.weight, w.scale, xq.scales_fp32() if fp8 else None, w.bias, act, gate, res, torch.float32)
    assert torch.allclose(y, ref, rtol=2 ** -7, atol=2 ** -7), (y - ref).abs().max()      # one rounding to bf16; fp32 sums


def test_output_rows_apart():
    torch.manual_seed(1)
    x = torch.randn(260, 192, device="cuda").to(torch.bfloat16)
    w = ops.LinearWeight.from_dense((torch.randn(320, 192, device="cuda") * 0.07).to(torch.bfloat16))
    for pitch in (328, 321):                              # rows on 16-byte boundaries, and not
        buf = torch.zeros(260, pitch, dtype=torch.bfloat16, device="cuda")
        ops.linear(x, w, out=buf[:, :320])
        assert torch.allclose(buf[:, :320].float(), x.float() @ w.weight.float().t(), rtol=2 ** -7, atol=2 ** -7)
        assert not buf[:, 320:].any()


def test_attention_into_rows_apart():
    torch.manual_seed(2)
    for t, h in ((257, 3), (600, 2)):
        q, k, v = (torch.randn(t, h, 128, device="cuda").to(torch.bfloat16) for _ in range(3))
        buf = torch.zeros(t, h * 128 + 24, dtype=torch.bfloat16, device="cuda")
        ops.attention(q, k, v, out=buf[:, 8:8 + h * 128])
        ref = R.attention(q, k, v)
        assert torch.allclose(buf[:, 8:8 + h * 128].float().reshape(t, h, 128), ref.float(), rtol=2e-2, atol=1e-2)
        assert not buf[:, :8].any() and not buf[:, 8 + h * 128:].any()


# a wave of 128 x 256 tiles and a few more: rows up to the line between a wave of whole tiles and ranges of K, and beyond it
@pytest.mark.parametrize("k,fp8", [(512, False), (12288, False), (12296, False), (512, True), (16384, True), (16512, True)])
def test_tail_after_a_full_wave(k, fp8):
    torch.manual_seed(k)
    m, n = 250, 19456
    x = torch.randn(m, k, device="cuda").to(torch.bfloat16)
    w = ops.LinearWeight.from_dense((torch.randn(n, k, device="cuda") * k ** -0.5).to(torch.bfloat16), fp8=fp8)
    xq = ops.quant_fp8_act(x) if fp8 else x
    y = ops.linear(xq, w).float()
    ref = R.linear(xq.data if fp8 else x, w.weight, w.scale, xq.scales_fp32() if fp8 else None, out_dtype=torch.float32)
    assert torch.allclose(y, ref, rtol=2 ** -7, atol=2 ** -7), (y - ref).abs().max()      # one rounding to bf16; fp32 sums


# 75 to 147 tiles of 128 features for few tokens: ranges of K in more than one wave, down to depths that leave no ranges
@pytest.mark.parametrize("m,n,k", [(5, 9600, 128), (64, 9596, 512), (33, 10240, 1152), (16, 9728, 896), (7, 18816, 4096), (128, 12288, 2048)])
@pytest.mark.parametrize("fp8", [False, True])
def test_few_tokens_more_than_half_a_wave(m, n, k, fp8):
    torch.manual_seed(m)
    x = torch.randn(m, k, device="cuda").to(torch.bfloat16)
    w = ops.LinearWeight.from_dense((torch.randn(n, k, device="cuda") * k ** -0.5).to(torch.bfloat16),
                                    torch.randn(n, device="cuda").to(torch.bfloat16), fp8=fp8)
    res = torch.randn(m, n, device="cuda").to(torch.bfloat16)
    xq = ops.quant_fp8_act(x) if fp8 else x
    y = ops.linear(xq, w, act="silu", residual=res).float()
    ref = R.linear(xq.data if fp8 else x, w.weight, w.scale, xq.scales_fp32() if fp8 else None, w.bias, "silu", None, res, torch.float32)
    assert torch.allclose(y, ref, rtol=2 ** -7, atol=2 ** -7), (y - ref).abs().max()      # one rounding to bf16; fp32 sums


@pytest.mark.parametrize("m,f,k", [(129, 23808, 64), (300, 15872, 136), (2177, 2688, 1024), (4737, 1280, 328)])
@pytest.mark.parametrize("act", ["silu", "gelu_tanh"])
def test_gated_tiles(m, f, k, act):
    torch.manual_seed(m)
    x = (torch.randn(m, k, device="cuda")).to(torch.bfloat16)
    w = ops.LinearWeight((torch.randn(2 * f, k, device="cuda") * 2 * k ** -0.5).to(torch.bfloat16))
    y, q = ops.linear_glu(x, w, act)
    ref = R.glu(x.float() @ w.weight.float().t(), act)
    assert q is None and torch.allclose(y.float(), ref, rtol=2 ** -7, atol=2 ** -8)      # fp32 sums, one rounding to bf16


@pytest.mark.parametrize("m,f,k", [(129, 23808, 128), (300, 15872, 640), (2177, 2688, 1024), (4737, 1280, 384)])
@pytest.mark.parametrize("act", ["silu", "gelu_tanh"])
def test_gated_tiles_fp8(m, f, k, act):
    if not ops.fp8_mx():
        pytest.skip("block scales in fp32")
    torch.manual_seed(m)
    w = ops.LinearWeight.from_dense((torch.randn(2 * f, k, device="cuda") * 2 * k ** -0.5).to(torch.bfloat16), fp8=True)
    x = ops.quant_fp8_act(torch.randn(m, k, device="cuda").to(torch.bfloat16))
    y, q = ops.linear_glu(x, w, act, emit_fp8=True, emit_bf16=False)
    ref = R.glu(R.linear(x.data.cpu(), w.weight.cpu(), w.scale.cpu(), x.scales_fp32().cpu(), out_dtype=torch.float32), act)
    assert y is None and q.data.shape == (m, f)
    got, s = R.dequant_fp8_act(q.data.cpu(), q.scales_fp32().cpu()), q.scales_fp32().cpu().repeat_interleave(128, 1)
    # half a step of e4m3 (2^-4 of a value, 2^-10 scales at least) and the rounding to bf16 ahead of it
    assert ((got - ref).abs() <= ref.abs() * (2 ** -4 + 2 ** -7) + s * 2 ** -10 + 2 ** -9).all()
    mx = ref.abs().reshape(m, -1, 128).amax(-1)
    assert (q.scales_fp32().cpu() * 448 * (1 + 2 ** -6) + 2 ** -9 >= mx).all() and (q.scales_fp32().cpu() * 448 <= 2 * (1 + 2 ** -6) * mx + 2 ** -8).all()


# products and attention that leave e4m3: the same bytes and scales as a quantisation of what they store otherwise
@pytest.mark.parametrize("m,n,k,q_from,lead", [(256, 9472, 2048, 0, 0), (300, 12416, 3072, 0, 256), (2049, 2432, 4096, 0, 0), (1651, 4224, 2048, 1408, 384), (4100, 1280, 4096, 1152, 128)])
@pytest.mark.parametrize("act", [None, "gelu_tanh"])
def test_quantised_product(m, n, k, q_from, lead, act):
    if not ops.fp8_mx():
        pytest.skip("block scales in fp32")
    torch.manual_seed(m)
    x = ops.quant_fp8_act(torch.randn(m, k, device="cuda").to(torch.bfloat16))
    w = ops.LinearWeight.from_dense((torch.randn(n, k, device="cuda") * k ** -0.5).to(torch.bfloat16), torch.randn(n, device="cuda").to(torch.bfloat16), fp8=True)
    y, q = ops.linear_quant(x, w, act=act, act_from=q_from if act else 0, q_from=q_from, lead=lead)
    ref = ops.linear(x, w, act=act, act_from=q_from if act else 0)
    assert (y is None) == (q_from == 0) and (y is None or torch.equal(y, ref[:, :q_from]))
    want = ops.quant_fp8_act(ref[:, q_from:].contiguous())
    assert torch.equal(q.data[:, lead:], want.data) and torch.equal(q.scales_fp32()[:, lead // 128:], want.scales_fp32())


def test_small_products_are_not_quantised_in_place():
    if not ops.fp8_mx():
        pytest.skip("block scales in fp32")
    w = ops.LinearWeight.from_dense(torch.randn(4096, 1024, device="cuda").to(torch.bfloat16), fp8=True)
    x = torch.randn(1000, 1024, device="cuda").to(torch.bfloat16)
    assert ops.linear_quant(ops.quant_fp8_act(x[:128]), w) is None and ops.linear_quant(x, w) is None
    assert ops.linear_quant(ops.quant_fp8_act(x), w, q_from=64) is None


@pytest.mark.parametrize("tq,tk,h,split,col", [(257, 256, 3, 257, 0), (600, 600, 2, 88, 128), (1000, 300, 1, 512, 0), (130, 777, 5, 130, 640)])
def test_quantised_attention(tq, tk, h, split, col):
    if not ops.attention_quant_fits(h, h, 128, tk):
        pytest.skip("attention leaves bf16 in this mode")
    torch.manual_seed(tq)
    q = torch.randn(tq, h, 128, device="cuda").to(torch.bfloat16)
    k, v = (torch.randn(tk, h, 128, device="cuda").to(torch.bfloat16) for _ in range(2))
    sizes = [split, tq - split] if split < tq else [tq]
    parts = [(ops.empty_fp8_act(r, h * 128 + col + 128 * i, "cuda"), r, col + 128 * i) for i, r in enumerate(sizes)]
    ops.attention_quant(q, k, v, parts)
    ref, at = ops.attention(q, k, v).reshape(tq, -1), 0
    for a, r, c in parts:
        want = ops.quant_fp8_act(ref[at:at + r].contiguous())
        assert torch.equal(a.data[:, c:c + h * 128], want.data) and torch.equal(a.scales_fp32()[:, c // 128:c // 128 + h], want.scales_fp32())
        at += r


# few tokens, more tiles than SMs: even shares of K groups, whose boundaries cut tiles into two pieces; rows of one group, ragged
# groups, features that end inside a tile, every epilogue, and the same again from the counters that the first launch left
@pytest.mark.parametrize("m,n,k", [(5, 19200, 640), (64, 28411, 1024), (17, 44416, 136), (128, 28672, 4096), (100, 24576, 1536), (33, 19100, 72), (1, 38528, 9216)])
@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("act", [None, "silu", "gelu_tanh", "tanh"])
def test_even_shares(m, n, k, fp8, act):
    torch.manual_seed(m)
    k = -(-k // 128) * 128 if fp8 else k
    x = torch.randn(m, k, device="cuda").to(torch.bfloat16)
    vec = lambda: torch.randn(n, device="cuda").to(torch.bfloat16) if act else None
    w = ops.LinearWeight.from_dense((torch.randn(n, k, device="cuda") * k ** -0.5).to(torch.bfloat16), vec(), fp8=fp8)
    gate = vec()
    res = torch.randn(m, n, device="cuda").to(torch.bfloat16) if act else None
    xq = ops.quant_fp8_act(x) if fp8 else x
    y = ops.linear(xq, w, act=act, act_from=8 if act == "tanh" else 0, gate=gate, residual=res)
    ref = R.linear(xq.data if fp8 else x, w.weight, w.scale, xq.scales_fp32() if fp8 else None, w.bias, act, gate, res, torch.float32,
                   act_from=8 if act == "tanh" else 0)
    assert torch.allclose(y.float(), ref, rtol=2 ** -7, atol=2 ** -7), (y.float() - ref).abs().max()      # one rounding to bf16; fp32 sums
    assert torch.equal(ops.linear(xq, w, act=act, act_from=8 if act == "tanh" else 0, gate=gate, residual=res), y)


# the two other operand types: s32 accumulators with row scales, and scales of 1x128 and 128x128 blocks, which a piece reads from the middle of
# a row of them on
@pytest.mark.parametrize("m,n,k", [(5, 19200, 640), (64, 28416, 1024), (17, 44416, 896), (100, 24576, 1536), (33, 19072, 512), (3, 38528, 4736)])
@pytest.mark.parametrize("int8", [True, False])
@pytest.mark.parametrize("act", [None, "gelu_tanh"])
def test_even_shares_other_types(m, n, k, int8, act):
    torch.manual_seed(m)
    x = torch.randn(m, k, device="cuda").to(torch.bfloat16)
    dense = (torch.randn(n, k, device="cuda") * k ** -0.5).to(torch.bfloat16)
    bias = torch.randn(n, device="cuda").to(torch.bfloat16) if act else None
    res = torch.randn(m, n, device="cuda").to(torch.bfloat16) if act else None
    if int8:
        w = ops.Int8Weight.from_dense(dense, bias)
        q, s = ops.quant_int8_act(x)
        run = lambda: ops.linear(x, w, act=act, residual=res)
        ref = (q.double() @ w.weight.double().T) * s.double()[:, None] * w.row_scale.double()[None]
    else:
        wq, wsc = R.quant_fp8_weight(dense)
        xq, xsc = R.quant_fp8_act(x)
        w = ops.LinearWeight(wq, wsc, bias)
        run = lambda: ops.linear(ops.Fp8Act(xq, xsc), w, act=act, residual=res)
        ref = R.linear(xq, wq, wsc, xsc, None, None, None, None, torch.float32).double()
    ref = ref + bias.double() if act else ref
    ref = torch.nn.functional.gelu(ref, approximate="tanh") + res.double() if act else ref
    y = run()
    assert torch.allclose(y.double(), ref, rtol=2 ** -7, atol=2 ** -7), (y.double() - ref).abs().max()      # one rounding to bf16; fp32 sums
    assert torch.equal(run(), y)


# Streams of one device share the scratch, so a product that does without it must leave it alone: few tokens and a last wave more than half
# full (above all with long rows), rows of too few K blocks to cut, and many tokens on CTA pairs
@pytest.mark.parametrize("m,n,k", [(6, 28672, 4096), (64, 28672, 4096), (128, 30720, 8192), (17, 29000, 4608), (33, 151936, 192), (5, 19200, 64), (300, 12288, 3072)])
@pytest.mark.parametrize("fp8", [False, True])
def test_whole_tiles_leave_the_scratch_alone(m, n, k, fp8):
    if fp8 and k % 128:
        pytest.skip("groups of 128")
    from hartsyinference_b200.ops import _native as N
    from hartsyinference_b200.ops import core
    torch.manual_seed(n)
    x = torch.randn(m, k, device="cuda").to(torch.bfloat16)
    w = ops.LinearWeight.from_dense((torch.randn(n, k, device="cuda") * k ** -0.5).to(torch.bfloat16), fp8=fp8)
    xq = ops.quant_fp8_act(x) if fp8 else x
    xs, ws = core._scale_ptrs(xq, w)
    xd = xq.data if fp8 else xq
    scratch = torch.zeros(64 << 20, dtype=torch.uint8, device="cuda")
    scratch[16384:] = 0xA5                           # behind the counters, which are zero between launches
    before, out = scratch.clone(), torch.empty(m, n, dtype=torch.bfloat16, device="cuda")
    N.check(N.lib().b200_gemm(xd.data_ptr(), w.weight.data_ptr(), out.data_ptr(), m, n, k, k, k, n, core._gemm_dtype(w), xs, ws, None, None, None, 0, 0,
                              scratch.data_ptr(), scratch.numel(), N.state(x.device).status.data_ptr(), N.stream()), "b200_gemm")
    assert torch.equal(scratch, before) and torch.equal(out, ops.linear(xq, w))
