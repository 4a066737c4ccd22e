"""Sampler kernel: rows decided by the entries near the maximum and rows that need the whole vocabulary, against the filters in
64 bits; the penalty inside the kernel against penalised scores."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _kept(x, k, p):
    """Sets of entries that top-k and then top-p keep, in 64 bits: an entry stays unless k entries are larger, and unless the mass of
    larger ones reaches p.  Also whether a row's top-p cut is further than 1e-5 from every entry's boundary."""
    n, v = x.shape
    s, order = x.sort(dim=1, descending=True)
    first = torch.searchsorted(-s, -s, right=False)          # entries strictly larger than each
    keep = (k.view(-1, 1) == 0) | (first < k.view(-1, 1))
    w = torch.where(keep, (s - s[:, :1]).exp(), torch.zeros_like(s))
    w = w / w.sum(1, keepdim=True)
    above = torch.cat([w.new_zeros(n, 1), w.cumsum(1)], 1).gather(1, first)
    safe = ((above - p.view(-1, 1)).abs() > 1e-5).all(1) | (p >= 1)
    keep &= (above < p.view(-1, 1)) | (p.view(-1, 1) >= 1)
    return torch.zeros(n, v, dtype=torch.bool, device=x.device).scatter_(1, order, keep), safe


@pytest.mark.parametrize("rows", [3, 150])                     # 1024 and 512 threads a row
@pytest.mark.parametrize("vocab", [1, 9, 2047, 2500, 32003, 128256])
@pytest.mark.parametrize("spread", [0.01, 3.0])                 # all entries near the maximum (the list overflows), and few
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_cuts_choices_and_logprobs(rows, vocab, spread, dtype):
    from tgi_b200.ops import cuda as K

    K.load()
    g = torch.Generator(device="cuda").manual_seed(rows + vocab)
    logits = (torch.randn(rows, vocab + 3, device="cuda", generator=g) * spread).to(dtype)[:, :vocab]      # unaligned rows
    if vocab % 2:
        logits = logits.contiguous()
    temp = torch.rand(rows, device="cuda", generator=g) + 0.5
    k = torch.tensor([0, 1, 40, 3000, vocab], device="cuda", dtype=torch.int32).repeat(rows)[:rows]
    p = torch.tensor([0.0, 0.5, 1.0, 0.9, 0.9999, 1.0], device="cuda").repeat(rows)[:rows]
    pen = torch.tensor([1.0, 1.3, 0.8], device="cuda").repeat(rows)[:rows]
    history = torch.randint(0, vocab, (rows, 65), device="cuda", generator=g)
    history[:, 50:] = 0
    history[0, 0] = vocab + 7                                  # outside the vocabulary: skipped
    sample = (torch.arange(rows, device="cuda") % 2).to(torch.uint8)
    seeds, steps = torch.arange(rows, device="cuda"), torch.full((rows,), 3, device="cuda", dtype=torch.int32)
    scores = K.penalties(logits, history, pen, None)
    ids, lps = K.fused_sample(logits, temp, k, p, sample, seeds, steps, history=history, repetition_penalty=pen)
    again, _ = K.fused_sample(scores, temp, k, p, sample, seeds, steps)
    assert torch.equal(ids, again)
    # the kernel multiplies by 1 / temperature in fp32
    x = (scores * (1 / temp).view(-1, 1)).double()
    keep, safe = _kept(x, k, p)
    assert (keep.gather(1, ids.view(-1, 1)).view(-1) | ~safe).all()
    want = x - torch.where(keep, x, torch.full_like(x, -torch.inf)).logsumexp(1, keepdim=True)
    # __expf and __logf: 2 ulp of fp32 plus 2^-21.4 absolute, on sums of up to 128k terms and scores up to 30
    assert ((lps - want.gather(1, ids.view(-1, 1)).view(-1)).abs()[safe] < 1e-4).all()
    top = x.max(1).values
    assert torch.equal(x.gather(1, ids.view(-1, 1)).view(-1)[sample == 0], top[sample == 0])


def test_rows_without_a_choice_and_rows_with_infinities():
    from tgi_b200.ops import cuda as K

    K.load()
    x = torch.randn(4, 1000, device="cuda")
    x[0] = -torch.inf
    x[1, :999] = -torch.inf
    x[2, 5] = torch.inf
    x[3, ::2] = -torch.inf
    p, sample = torch.full((4,), 0.7, device="cuda"), torch.ones(4, device="cuda", dtype=torch.uint8)
    seeds, steps = torch.arange(4, device="cuda"), torch.zeros(4, device="cuda", dtype=torch.int32)
    for top_p in (None, p):
        ids, lps = K.fused_sample(x, None, None, top_p, sample, seeds, steps)
        assert ids[0].item() == 0 and ids[1].item() == 999 and ids[3].item() % 2 == 1
        assert abs(lps[1].item()) < 1e-6 and torch.isfinite(lps[3])
