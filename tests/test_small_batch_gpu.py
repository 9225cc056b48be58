"""Small-batch forms: K ranges summed by the norm and the rotary kernel, argmax in 16-byte reads."""
from dataclasses import replace

import pytest
import torch

from hartsyinference_b200 import ops
from hartsyinference_b200.engine.sampling import SamplingParams, sample_row
from hartsyinference_b200.models.llm import config as C
from hartsyinference_b200.models.llm.transformer import DecoderModel, ForwardBatch
from hartsyinference_b200.ops import reference as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [5, 17, 64, 128])
@pytest.mark.parametrize("n,k,fp8", [(896, 4864, False), (8192, 1024, False), (1024, 3072, True)])
def test_norm_adds_the_ranges(m, n, k, fp8):
    torch.manual_seed(m)
    x = torch.randn(m, k, device="cuda").to(torch.bfloat16)
    w = ops.LinearWeight.from_dense((torch.randn(n, k, device="cuda") * k ** -0.5).to(torch.bfloat16), fp8=fp8)
    res, g = (torch.randn(*s, device="cuda").to(torch.bfloat16) for s in ((m, n), (n,)))
    part = ops.linear(x, w, defer=True)
    assert isinstance(part, ops.core.SplitSum) and part.splits > 1
    y, h, q = ops.norm(part, g, residual=res, emit_fp8=True)
    y2, h2, q2 = ops.norm(ops.linear(x, w), g, residual=res, emit_fp8=True)
    # the same addends in the same order
    assert torch.equal(h, h2) and torch.equal(y, y2) and torch.equal(q.data, q2.data)


@pytest.mark.parametrize("m", [5, 33])
@pytest.mark.parametrize("d,style", [(64, 0), (128, 1), (96, 0)])
def test_rotary_adds_ranges_and_bias(m, d, style):
    torch.manual_seed(m + d)
    hq, hkv, k = 6, 2, 1024
    n = (hq + 2 * hkv) * d
    x = torch.randn(m, k, device="cuda").to(torch.bfloat16)
    w = ops.LinearWeight.from_dense((torch.randn(n, k, device="cuda") * k ** -0.5).to(torch.bfloat16), torch.randn(n, device="cuda").to(torch.bfloat16))
    pos = torch.randint(0, 3000, (m,), dtype=torch.int32, device="cuda")
    part = ops.linear(x, w, defer=True, defer_bias=True)
    assert isinstance(part, ops.core.SplitSum)
    got = ops.rope_kv(part, pos, hq, hkv, d, style=style, want_kv=True)
    ref = ops.rope_kv(ops.linear(x, w), pos, hq, hkv, d, style=style, want_kv=True)
    for a, b in zip(got, ref):
        assert torch.equal(a, b)


@pytest.mark.parametrize("m,n,k", [(5, 896, 4864), (64, 1024, 1024), (128, 9600, 4096), (17, 9600, 2048)])
def test_ranges_outlive_other_products(m, n, k):
    """A second product that is cut along K, between the first one and its consumer: the ranges are the consumer's."""
    torch.manual_seed(n)
    x, x2 = (torch.randn(m, k, device="cuda").to(torch.bfloat16) for _ in range(2))
    w, w2 = (ops.LinearWeight((torch.randn(n, k, device="cuda") * k ** -0.5).to(torch.bfloat16)) for _ in range(2))
    want, want2 = ops.norm(ops.linear(x, w))[0], ops.norm(ops.linear(x2, w2))[0]
    part = ops.linear(x, w, defer=True)
    assert isinstance(part, ops.core.SplitSum)
    assert torch.equal(ops.norm(ops.linear(x2, w2))[0], want2)
    assert torch.equal(ops.norm(ops.linear(x2, w2, defer=True))[0], want2)
    assert torch.equal(ops.norm(part)[0], want)


@pytest.mark.parametrize("vocab", [1, 7, 8, 1025, 32768, 32777, 151936])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_argmax_takes_the_first_of_equals(vocab, dtype):
    torch.manual_seed(vocab)
    x = torch.randn(9, vocab + 8, device="cuda").to(dtype)[:, :vocab]
    x[1] = 0.0
    if vocab > 7:
        x[2, vocab - 1] = x[2, vocab // 2] = 60.0
        x[3, vocab - 1] = 60.0
    want = torch.tensor([int((r == r.max()).nonzero()[0]) for r in x.cpu()])
    for y in (x, x.contiguous(), x[:, :]):
        assert torch.equal(ops.argmax(y).cpu().long(), want)
    many = x.repeat(40, 1) if vocab < 40000 else x                     # more rows than processors: smaller blocks
    assert torch.equal(ops.argmax(many).cpu().long(), want.repeat(many.shape[0] // 9))


@pytest.mark.parametrize("vocab,pitch", [(1, 8), (8, 8), (1025, 1032), (1025, 1033), (32777, 32784), (151936, 151936)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_argmax_of_rows_without_a_finite_value(vocab, pitch, dtype):
    x = torch.full((3, pitch), float("-inf"), device="cuda", dtype=dtype)[:, :vocab]
    x[1, vocab - 1] = torch.finfo(dtype).min
    assert ops.argmax(x).tolist() == [0, vocab - 1, 0]
    p = SamplingParams(greedy=True, logits_mask=lambda history: torch.zeros(vocab, dtype=torch.bool))
    lg = torch.randn(vocab)
    assert sample_row(lg.cuda(), p, [], None) == sample_row(lg, p, [], None) == 0      # a grammar that allows nothing


def test_gated_product_of_no_rows():
    w = ops.LinearWeight(torch.randn(512, 256, device="cuda").to(torch.bfloat16))
    y, q = ops.linear_glu(torch.empty(0, 256, device="cuda", dtype=torch.bfloat16), w)
    assert tuple(y.shape) == (0, 256) and q is None


# the product that norms its input and rotates its output: depths that leave lanes idle, heads with and without an unrotated rest
@pytest.mark.parametrize("m", [1, 2, 3, 4])
@pytest.mark.parametrize("k,hq,hkv,d,rot,style,bias", [(896, 14, 2, 64, 64, 0, True), (512, 4, 4, 96, 96, 1, False), (2056, 8, 2, 128, 64, 0, True),
                                                      (128, 2, 1, 64, 32, 1, False), (64, 2, 2, 32, 0, 0, False)])
def test_one_launch_of_norm_projection_and_rotation(m, k, hq, hkv, d, rot, style, bias):
    torch.manual_seed(k + m)
    bf = torch.bfloat16
    x = torch.randn(m, k, device="cuda").to(bf)
    nw = (1 + 0.1 * torch.randn(k, device="cuda")).to(bf)
    n = (hq + 2 * hkv) * d
    w = ops.LinearWeight((torch.randn(n, k, device="cuda") * k ** -0.5).to(bf), bias=torch.randn(n, device="cuda").to(bf) if bias else None)
    pos = torch.randint(0, 30000, (m,), device="cuda", dtype=torch.int32)
    inv = R.rope_inv_freq(max(rot, 2), 10000.0, torch.device("cuda")).float()
    slots = torch.tensor([5, -1, 17, 40][:m], device="cuda")
    caches = [torch.zeros(2, 3, hkv, 16, d, dtype=bf, device="cuda") for _ in range(2)]
    q = ops.norm_qkv_few(x, nw, w, pos, hq, hkv, d, k_cache=caches[0][0], v_cache=caches[0][1], slot_mapping=slots, rot=rot, inv_freq=inv, style=style, ahead=(w,))
    h = ops.norm(x, nw)[0]
    y = (h.float() @ w.weight.float().t() + (w.bias.float() if bias else 0)).to(bf)
    ref = ops.rope_kv(y, pos, hq, hkv, d, k_cache=caches[1][0], v_cache=caches[1][1], slot_mapping=slots, rot=rot, inv_freq=inv, style=style)[0]
    # the sums of k products in fp32 differ in order, so a value may round to the neighbouring bf16 in front of the rotation and behind it
    for a, b in ((q, ref), (caches[0], caches[1])):
        assert (a.float() - b.float()).abs().max() <= 2 ** -6 * max(1.0, b.float().abs().max().item())
        assert (a.float() - b.float()).norm() <= 2e-3 * b.float().norm() + 1e-6


@pytest.mark.parametrize("m,f,k", [(1, 4864, 896), (2, 40, 512), (3, 1000, 2056), (4, 13, 64), (1, 14336, 4096), (1, 8, 8192)])
@pytest.mark.parametrize("act", ["silu", "gelu_tanh"])
def test_one_launch_of_norm_and_gated_product(m, f, k, act):
    torch.manual_seed(f)
    bf = torch.bfloat16
    x = torch.randn(m, k, device="cuda").to(bf)
    nw = (1 + 0.1 * torch.randn(k, device="cuda")).to(bf)
    w = ops.LinearWeight((torch.randn(2 * f, k, device="cuda") * k ** -0.5).to(bf))
    y = ops.norm_glu_few(x, nw, w, act, weight_plus_one=f == 40, ahead=(w, w))
    ref = R.glu(ops.norm(x, nw, weight_plus_one=f == 40)[0].float() @ w.weight.float().t(), act)
    assert torch.allclose(y.float(), ref, rtol=2 ** -7, atol=2 ** -8)      # fp32 sums, one rounding to bf16


def test_one_token_through_the_stack():
    for preset in ("qwen2.5-0.5b", "llama-3-8b"):
        cfg = replace(C.PRESETS[preset], num_layers=2, vocab_size=512)
        model = DecoderModel(cfg, "cuda")
        model.random_init(seed=1)
        model.alloc_kv(4, 16)
        model.kv_cache.normal_()
        dev = lambda *v, dtype=torch.int32: torch.tensor(v, dtype=dtype, device="cuda")
        batch = ForwardBatch(tokens=dev(7), positions=dev(40), slot_mapping=dev(2 * 16 + 8, dtype=torch.int64), block_table=dev(0, 1, 2).reshape(1, 3),
                             kv_lens=dev(41), is_decode=True, max_kv_len=48)
        assert model._few_ok(batch, torch.zeros(1, cfg.hidden_size, dtype=torch.bfloat16, device="cuda"))
        before = model.kv_cache.clone()
        y, cache = model.forward_hidden(batch), model.kv_cache.clone()
        model.kv_cache.copy_(before)
        model._few_ok = lambda *a: False
        ref = model.forward_hidden(batch)
        # two layers of bf16 roundings that fall differently (one sum is no longer rounded ahead of the residual add)
        assert (y.float() - ref.float()).norm() <= 2e-2 * ref.float().norm()
        assert (cache.float() - model.kv_cache.float()).norm() <= 2e-3 * model.kv_cache.float().norm()


# prompts through a plain stack: the same kernels whether the library or the loop of ops walks the layers, at the sizes where their choices
# change (handful, ranges left unsummed, pair tiles, either attention kernel)
@pytest.mark.parametrize("preset", ["qwen2.5-0.5b", "llama-3-8b"])
@pytest.mark.parametrize("lens,held", [([1], 0), ([3], 5), ([17, 5, 7], 0), ([100, 28], 30), ([129], 0), ([700, 64, 260], 16)])
def test_prompts_by_the_library_and_by_ops(preset, lens, held):
    cfg = replace(C.PRESETS[preset], num_layers=2, vocab_size=512)
    model = DecoderModel(cfg, "cuda")
    model.random_init(seed=2)
    per = [(n + held + 15) // 16 for n in lens]
    model.alloc_kv(sum(per), 16)
    model.kv_cache.normal_()
    g = torch.Generator().manual_seed(3)
    order, table, at = torch.randperm(sum(per), generator=g).to(torch.int32), torch.zeros(len(lens), max(per), dtype=torch.int32), 0
    for i, c in enumerate(per):
        table[i, :c] = order[at:at + c]
        at += c
    pos = torch.cat([torch.arange(held, held + n) for n in lens])
    seq = torch.repeat_interleave(torch.arange(len(lens)), torch.tensor(lens))
    slots = table[seq, pos // 16].long() * 16 + pos % 16
    dev = lambda t, dt=torch.int32: torch.as_tensor(t).to(dt).cuda()
    batch = ForwardBatch(tokens=dev(torch.randint(0, 512, (sum(lens),), generator=g)), positions=dev(pos), slot_mapping=dev(slots, torch.int64), block_table=dev(table),
                         kv_lens=dev([n + held for n in lens]), is_decode=False, cu_q=dev(torch.tensor([0] + lens).cumsum(0)), max_q_len=max(lens),
                         max_kv_len=max(lens) + held)
    assert model._plain_stack(batch, torch.zeros(1, cfg.hidden_size, dtype=torch.bfloat16, device="cuda"))
    before = model.kv_cache.clone()
    y, cache = model.forward_hidden(batch), model.kv_cache.clone()
    model.kv_cache.copy_(before)
    model._prompt_layers = lambda *a: None
    assert torch.equal(model.forward_hidden(batch), y) and torch.equal(model.kv_cache, cache)
