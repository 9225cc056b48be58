"""Small-batch forms: K ranges summed by the norm and the rotary kernel, argmax in 16-byte reads."""
import pytest
import torch

from hartsyinference_b200 import ops
from hartsyinference_b200.engine.sampling import SamplingParams, sample_row

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
