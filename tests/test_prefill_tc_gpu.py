"""Paged causal prefill on the tcgen05 kernel against the fp32 statement, at the edges of its tiles and pages."""
import pytest
import torch

from hartsyinference_b200 import ops
from hartsyinference_b200.ops import reference as R

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hq,hkv", [(8, 2), (6, 2), (4, 4)])          # groups of 4 (heads in pairs), 3 and 1 (tiles in pairs)
@pytest.mark.parametrize("page,lens", [
    (16, [(1, 1), (127, 127), (128, 128), (129, 129), (300, 300)]),     # (query tokens, keys): ends of query tiles
    (16, [(1, 128), (1, 129), (2, 257), (64, 500), (257, 1000)]),       # chunks behind a cached prefix, ends of key tiles
    (8, [(17, 41), (130, 136)]), (32, [(256, 256), (33, 97)]), (64, [(5, 5), (200, 391)])])
@pytest.mark.parametrize("most", [1 << 16, None])                     # keys that a sequence may have: tcgen05 at any size, or as sizes have it
def test_against_fp32(hq, hkv, page, lens, most):
    torch.manual_seed(len(lens) + page + hq)
    d = 128
    need = [(n + page - 1) // page for _, n in lens]
    pages = sum(need) + 3
    kc = torch.full((pages, hkv, page, d), float("nan"), dtype=torch.bfloat16, device="cuda")      # rows nobody wrote
    vc = kc.clone()
    order = torch.randperm(pages)[:sum(need)]
    table = torch.full((len(lens), max(need) + 1), pages - 1, dtype=torch.int32)
    keys, values, at = [], [], 0
    for i, (_, n) in enumerate(lens):
        own = order[at:at + need[i]]
        at += need[i]
        table[i, :need[i]] = own.to(torch.int32)
        k, v = (torch.randn(n, hkv, d).to(torch.bfloat16) for _ in range(2))
        keys.append(k)
        values.append(v)
        for t in range(n):
            kc[own[t // page], :, t % page] = k[t].cuda()
            vc[own[t // page], :, t % page] = v[t].cuda()
    q_lens = [a for a, _ in lens]
    q = torch.randn(sum(q_lens), hq, d).to(torch.bfloat16)
    cu = torch.tensor([0] + q_lens).cumsum(0).to(torch.int32)
    out = ops.attn_prefill_paged(q.cuda(), kc, vc, table.cuda(), torch.tensor([n for _, n in lens], dtype=torch.int32, device="cuda"),
                                 cu.cuda(), max(q_lens), max_kv_len=most).float().cpu()
    for i in range(len(lens)):
        ref = R.attention(q[cu[i]:cu[i + 1]], keys[i], values[i], causal=True).float()
        got = out[cu[i]:cu[i + 1]]
        # probabilities and outputs are bf16: 2^-9 each of values below the largest of a few normal ones
        assert torch.allclose(got, ref, rtol=2e-2, atol=2e-2), (i, (got - ref).abs().max())
        assert (got - ref).norm() < 5e-3 * ref.norm()
