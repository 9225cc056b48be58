"""Products of one to four tokens with bf16 weights at the edges of rows per warp, shared rows and depth."""
import pytest
import torch

from hartsyinference_b200 import ops
from hartsyinference_b200.ops import reference as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("m", [1, 2, 3, 4])
@pytest.mark.parametrize("n,k", [(1, 8), (7, 264), (896, 4864), (1152, 896), (4097, 512), (8193, 1032), (3072, 15360)])
@pytest.mark.parametrize("act,act_from", [(None, 0), ("silu", 0), ("gelu_tanh", 5)])
def test_against_fp32(m, n, k, act, act_from):
    torch.manual_seed(n + m)
    x = torch.randn(m, k + 8, device="cuda").to(torch.bfloat16)[:, :k]
    w = ops.LinearWeight((torch.randn(n, k, device="cuda") * k ** -0.5).to(torch.bfloat16), None, torch.randn(n, device="cuda").to(torch.bfloat16))
    gate, res = torch.randn(n, device="cuda").to(torch.bfloat16), torch.randn(m, n, device="cuda").to(torch.bfloat16)
    y = ops.linear(x, w, act=act, act_from=act_from, gate=gate, residual=res).float()
    ref = R.linear(x, w.weight, None, None, w.bias, act, gate, res, torch.float32, act_from=act_from)
    assert torch.allclose(y, ref, rtol=2 ** -7, atol=2 ** -8)             # one rounding to bf16, fp32 sums
    out = torch.zeros(m, n + 3, dtype=torch.bfloat16, device="cuda")
    ops.linear(x, w, out=out[:, :n], defer=True)
    assert torch.allclose(out[:, :n].float(), R.linear(x, w.weight, bias=w.bias, out_dtype=torch.float32), rtol=2 ** -7, atol=2 ** -8)
    assert not out[:, n:].any()


def test_values_that_are_not_finite_stay_where_they_are():
    x = torch.ones(2, 264, device="cuda", dtype=torch.bfloat16)
    x[1, 263] = float("inf")
    w = torch.ones(9, 264, device="cuda", dtype=torch.bfloat16)
    w[3, 0] = float("nan")
    y = ops.linear(x, ops.LinearWeight(w))
    assert torch.isnan(y[0, 3]) and torch.isfinite(y[0, [0, 1, 2, 4, 5, 6, 7, 8]]).all()
    assert torch.isinf(y[1, [0, 1, 2, 4, 5, 6, 7, 8]]).all()


@pytest.mark.parametrize("m", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("f,k", [(8, 8), (4864, 896), (4104, 264), (1000, 4096)])
@pytest.mark.parametrize("act", ["silu", "gelu_tanh"])
def test_gated_product(m, f, k, act):
    torch.manual_seed(f + m)
    x = torch.randn(m, k, device="cuda").to(torch.bfloat16)
    w = ops.LinearWeight((torch.randn(2 * f, k, device="cuda") * k ** -0.5).to(torch.bfloat16))
    y, q = ops.linear_glu(x, w, act)
    ref = R.glu(x.float() @ w.weight.float().t(), act)
    assert q is None and torch.allclose(y.float(), ref, rtol=2 ** -6, atol=2 ** -8)      # five tokens round both halves first
