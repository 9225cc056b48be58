"""Row kernels at the sizes where their launch shapes and vector forms change, against the fp32 statements."""
import pytest
import torch

from hartsyinference_b200 import ops
from hartsyinference_b200.ops import reference as R

pytestmark = pytest.mark.gpu


def _rand(*shape, scale=1.0):
    return (torch.randn(*shape, device="cuda") * scale).to(torch.bfloat16)


@pytest.mark.parametrize("rows,dim", [(1, 8), (296, 8192), (297, 8192), (297, 2048), (297, 2040), (5, 16384), (300, 12288)])
@pytest.mark.parametrize("layernorm", [False, True])
def test_norm_shapes(rows, dim, layernorm):
    torch.manual_seed(dim)
    x, res, w, b = _rand(rows, dim), _rand(rows, dim), _rand(dim), _rand(dim)
    mod = _rand(2, 2 * dim + 4, scale=0.3)            # rows of the modulation that are not on 16-byte boundaries
    shift, scale = mod[:, 1:dim + 1], mod[:, dim + 2:2 * dim + 2]
    fp8 = dim % 128 == 0
    y, h, q = ops.norm(x, w, bias=b, residual=res, shift=shift, scale=scale, rows_per_batch=(rows + 1) // 2, eps=1e-5,
                       layernorm=layernorm, emit_fp8=fp8)
    yr, hr = R.norm(x.cpu(), w.cpu(), b.cpu(), res.cpu(), shift.cpu(), scale.cpu(), (rows + 1) // 2, 1e-5, layernorm, False)
    assert torch.equal(h.cpu(), hr)
    assert torch.allclose(y.float().cpu(), yr, rtol=2 ** -7, atol=2 ** -7)      # one rounding to bf16 and the row's sums
    if fp8:
        got = R.dequant_fp8_act(q.data, q.scales_fp32())
        assert (got - y.float()).norm() < 0.04 * y.float().norm()                  # half a step of e4m3 is 2^-4 of a value


@pytest.mark.parametrize("rows,f", [(1, 128), (3, 4864), (593, 2048), (4736, 256), (4737, 264)])
@pytest.mark.parametrize("act", ["silu", "gelu_tanh"])
def test_glu_shapes(rows, f, act):
    torch.manual_seed(f)
    x = _rand(rows, 2 * f, scale=3.0)
    fp8 = f % 128 == 0
    y, q = ops.glu(x, act, emit_fp8=fp8)
    ref = R.glu(x.cpu(), act)
    assert torch.allclose(y.float().cpu(), ref, rtol=2 ** -7, atol=1e-5)
    if fp8:
        again = ops.quant_fp8_act(y)
        assert torch.equal(q.data, again.data) and torch.equal(q.scales_fp32(), again.scales_fp32())


@pytest.mark.parametrize("rows,dim,pitch", [(1, 128, 128), (7, 384, 512), (1200, 2048, 2056), (4737, 128, 128)])
def test_fp8_quantisation_shapes(rows, dim, pitch):
    torch.manual_seed(rows)
    x = _rand(rows, pitch)[:, :dim]
    q = ops.quant_fp8_act(x)
    qr, sr = R.quant_fp8_act(x.cpu(), pow2=q.sf is not None)
    assert torch.equal(q.data.cpu(), qr) and torch.equal(q.scales_fp32().cpu(), sr)


@pytest.mark.parametrize("tokens", [1, 5, 1187])
@pytest.mark.parametrize("d,rot,style", [(16, 16, 0), (32, 16, 1), (64, 64, 0), (64, 32, 1), (128, 128, 1), (128, 64, 0), (256, 256, 0), (96, 96, 0), (128, 8, 1)])
@pytest.mark.parametrize("norm", [False, True])
def test_rotary_and_cache_write(tokens, d, rot, style, norm):
    torch.manual_seed(tokens + d)
    hq, hkv, page = 6, 2, 16
    qkv = _rand(tokens, (hq + 2 * hkv) * d)
    pos = torch.randint(0, 5000, (tokens,), dtype=torch.int32, device="cuda")
    pages = tokens // page + 2
    slots = torch.randperm(pages * page)[:tokens].to("cuda")
    slots[0] = -1                                                     # a row that is not stored
    kc = torch.zeros(pages, hkv, page, d, dtype=torch.bfloat16, device="cuda")
    vc = kc.clone()
    w = [_rand(d) if norm else None for _ in range(2)]
    inv = R.rope_inv_freq(rot, 1e4, "cuda")
    q, k, v = ops.rope_kv(qkv, pos, hq, hkv, d, k_cache=kc, v_cache=vc, slot_mapping=slots, rot=rot, inv_freq=inv, style=style,
                          q_norm_w=w[0], k_norm_w=w[1], want_kv=True)
    kr, vr = torch.zeros_like(kc).cpu(), torch.zeros_like(kc).cpu()
    cpu = [None if t is None else t.cpu() for t in w]
    qr, k2, v2 = ops.rope_kv(qkv.cpu(), pos.cpu(), hq, hkv, d, k_cache=kr, v_cache=vr, slot_mapping=slots.cpu(), rot=rot, inv_freq=inv.cpu(),
                             style=style, q_norm_w=cpu[0], k_norm_w=cpu[1], want_kv=True)
    for got, ref in ((q, qr), (k, k2), (v, v2), (kc, kr), (vc, vr)):
        assert torch.allclose(got.float().cpu(), ref.float(), rtol=2 ** -6, atol=2 ** -6)


@pytest.mark.parametrize("tokens,hq,hkv,d", [(1, 2, 2, 32), (77, 3, 1, 64), (130, 24, 24, 128), (9, 5, 5, 256), (33, 4, 4, 48), (3, 66, 2, 128)])
@pytest.mark.parametrize("row_norm", [False, True])
def test_dit_qkv_forms(tokens, hq, hkv, d, row_norm):
    torch.manual_seed(tokens)
    width = (hq + 2 * hkv) * d
    x = _rand(tokens, width + 64)[:, :width]
    wq, wk = (_rand(hq * d), _rand(hkv * d)) if row_norm else (_rand(d), _rand(d))
    ang = torch.randn(tokens, d // 2, device="cuda")
    out = tuple(torch.empty(tokens + 2, h, d, dtype=torch.bfloat16, device="cuda")[2:] for h in (hq, hkv, hkv))
    got = ops.dit_qkv(x, hq, hkv, d, q_norm_w=wq, k_norm_w=wk, cos=ang.cos(), sin=ang.sin(), row_norm=row_norm, out=out)
    ref = ops.dit_qkv(x.cpu(), hq, hkv, d, q_norm_w=wq.cpu(), k_norm_w=wk.cpu(), cos=ang.cos().cpu(), sin=ang.sin().cpu(), row_norm=row_norm)
    for g, o, r in zip(got, out, ref):
        assert g.data_ptr() == o.data_ptr()
        assert torch.allclose(g.float().cpu(), r.float(), rtol=2 ** -6, atol=2 ** -6)


@pytest.mark.parametrize("rows,f", [(1, 40), (5, 64), (1183, 64), (1185, 72), (2369, 128), (9473, 384), (37889, 128)])
def test_narrow_rows_share_a_block(rows, f):
    torch.manual_seed(rows)
    x, n8 = _rand(rows, 2 * f, scale=3.0), f % 128 == 0
    y, q = ops.glu(x, "silu", emit_fp8=n8)
    assert torch.allclose(y.float().cpu(), R.glu(x.cpu(), "silu"), rtol=2 ** -7, atol=1e-5)
    if n8:
        again = ops.quant_fp8_act(y)
        qr, sr = R.quant_fp8_act(y.cpu(), pow2=q.sf is not None)
        assert torch.equal(q.data, again.data) and torch.equal(q.scales_fp32(), again.scales_fp32())
        assert torch.equal(again.data.cpu(), qr) and torch.equal(again.scales_fp32().cpu(), sr)
