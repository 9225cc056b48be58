"""The sampler's row-in-registers form: vocabularies at the ends of its sizes, ties, infinities, one value of mass."""
import pytest
import torch

from hartsyinference_b200 import ops
from hartsyinference_b200.ops import reference as R

pytestmark = pytest.mark.gpu


def _sample(logits, t, k, p, mp, seed=0):
    n = logits.shape[0]
    full = lambda v, dt: torch.full((n,), v, dtype=dt, device="cuda")
    return ops.sample_tokens(logits, full(t, torch.float32), full(k, torch.int32), full(p, torch.float32), full(mp, torch.float32),
                             torch.arange(n, device="cuda") + seed, full(3, torch.int64))


@pytest.mark.parametrize("vocab", [1, 2, 511, 4097, 32768, 32769, 65537, 131073, 163841, 262144, 262145])
@pytest.mark.parametrize("t,k,p,mp", [(0.8, 40, 0.9, 0.0), (1.0, 0, 0.95, 0.05), (1.3, 0, 0.0, 0.0)])
def test_kept_set(vocab, t, k, p, mp):
    torch.manual_seed(vocab)
    logits = torch.randn(5, vocab, device="cuda") * 3
    tok = _sample(logits, t, k, p, mp)
    for r in range(5):
        assert bool(R.sampling_keep_mask(logits[r], t, k, p, mp)[int(tok[r])])
    assert torch.equal(_sample(logits, 0.0, k, p, mp), logits.argmax(-1).to(torch.int32))


def test_draw_follows_the_prefix_sums():
    """The draw is the first index whose prefix mass passes u: found again in 64 bits from the same uniform number."""
    torch.manual_seed(5)
    n, vocab = 64, 50257
    logits = torch.randn(n, vocab, device="cuda") * 2
    tok = _sample(logits, 1.0, 0, 0.0, 0.0, seed=11).tolist()
    mask = (1 << 64) - 1
    for r in range(n):
        z = (r + 11 + 0x9E3779B97F4A7C15 * 4) & mask
        z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & mask
        z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & mask
        u = ((z ^ (z >> 31)) >> 40) / 2 ** 24
        w = torch.exp((logits[r] - logits[r].max()).double())
        c = w.cumsum(0)
        lo = float(c[tok[r] - 1]) if tok[r] else 0.0
        # weights are fp32 exponentials (2^-21 relative at these arguments)
        assert lo - 1e-5 * float(c[-1]) <= u * float(c[-1]) <= float(c[tok[r]]) + 1e-5 * float(c[-1])


def test_ties_and_infinities():
    x = torch.zeros(4, 40000, device="cuda")
    x[0, 39999] = x[0, 123] = 9.0
    x[1] = float("-inf")
    x[1, 777] = 1.0
    x[2] = float("-inf")
    x[3, 5] = float("inf")
    x[3, 30000] = float("inf")
    assert _sample(x, 0.0, 0, 0.0, 0.0).tolist() == [123, 777, 0, 5]
    tok = _sample(x, 0.7, 50, 0.9, 0.1).tolist()
    assert tok[0] in (123, 39999) and tok[1:] == [777, 0, 5]
    assert set(_sample(x[:1].repeat(200, 1).contiguous(), 1.0, 1, 0.0, 0.0).tolist()) == {123, 39999}     # ties at the k-th value all stay


@pytest.mark.parametrize("rows,vocab", [(300, 32000), (300, 8193), (160, 5000)])
def test_many_rows_as_few(rows, vocab):
    """Batches that a block per row is faster for, against the same rows a few at a time and the sampler's statement."""
    torch.manual_seed(rows)
    logits = torch.randn(rows, vocab, device="cuda") * 3
    ids = torch.arange(rows, device="cuda")
    col = lambda values, dt: torch.tensor(values, dtype=dt, device="cuda").repeat((rows + 5) // 6)[:rows]
    args = (col([0.0, 0.8, 1.0, 0.7, 1.3, 1.0], torch.float32), col([0, 40, 0, 50, 0, 1], torch.int32), col([0.9, 0.95, 0.9, 0.0, 1.0, 0.0], torch.float32),
            col([0.0, 0.0, 0.05, 0.0, 0.1, 0.0], torch.float32), ids, ids * 3)
    tok = ops.sample_tokens(logits, *args)
    few = torch.cat([ops.sample_tokens(logits[i:i + 4], *(a[i:i + 4] for a in args)) for i in range(0, rows, 4)])
    greedy = args[0] <= 0
    assert torch.equal(tok[greedy], logits[greedy].argmax(-1).to(torch.int32))
    for r in range(rows):
        if not greedy[r]:
            assert bool(R.sampling_keep_mask(logits[r], *(float(a[r]) if a.is_floating_point() else int(a[r]) for a in args[:4]))[int(tok[r])])
    assert torch.equal(tok, few)      # both forms sum masses in 2^-40: a row's token does not depend on its batch


@pytest.mark.parametrize("t,k,p,mp", [(1.0, 0, 0.0, 0.0), (1.0, 0, 0.9, 0.0), (0.7, 20000, 0.95, 0.3)])
def test_flat_rows_of_a_large_batch(t, k, p, mp):
    """Tokens of 1e-5 each, where sums that round differ from one form to the other draw different tokens."""
    torch.manual_seed(7)
    logits = (torch.randn(1000, 100000, device="cuda") * 0.1).to(torch.bfloat16)
    few = torch.cat([_sample(logits[i:i + 8], t, k, p, mp, seed=i) for i in range(0, 1000, 8)])
    assert torch.equal(_sample(logits, t, k, p, mp), few)


# batches that go one block per row, and the same rows a few at a time, which go a cluster per row: the walk over runs of bins ends in
# the first and the last run, in a bin that many values share, and nowhere
@pytest.mark.parametrize("vocab", [2048, 4096, 16384])
@pytest.mark.parametrize("t,k,p,mp", [(0.8, 50, 0.9, 0.05), (1.0, 1, 0.0, 0.0), (1.0, -1, 0.999999, 0.0), (0.7, 0, 1e-6, 0.0), (1.0, -1, 0.5, 1.0), (0.05, 0, 0.97, 0.0)])
def test_blocks_and_clusters_draw_the_same(vocab, t, k, p, mp):
    torch.manual_seed(vocab + 1)
    x = torch.randn(160, vocab, device="cuda") * torch.linspace(0.01, 20, 160, device="cuda")[:, None]
    x[3] = 1.5
    x[4] = (torch.arange(vocab, device="cuda") % 7).float()
    x[5, 1:] = float("-inf")
    x[6] -= 50 * (torch.arange(vocab, device="cuda") % 2048 > 3)
    k = vocab - 1 if k < 0 else k
    many = _sample(x, t, k, p, mp)
    few = torch.cat([_sample(x[i:i + 8], t, k, p, mp, seed=i) for i in range(0, 160, 8)])
    assert torch.equal(many, few)
