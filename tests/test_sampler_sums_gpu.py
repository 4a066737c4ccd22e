"""Sampler kernel: what a row gives depends on nothing but the row: not on the signs of zeros among the listed entries, on the other
rows, on where it lies in memory, nor on the order in which penalised ids are met; histories on both sides of the list's size, NaN."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def _params(rows, cut):
    full = lambda v, dt=torch.float32: torch.full((rows,), v, device="cuda", dtype=dt)
    kw = {"none": {}, "top_p": {"top_p": full(0.9)}, "flat_p": {"top_p": full(0.9999)}, "top_k": {"top_k": full(50, torch.int32)},
          "both": {"top_k": full(50, torch.int32), "top_p": full(0.8)}, "typical": {"typical_p": full(0.8)},
          "all": {"top_k": full(5000, torch.int32), "top_p": full(0.95), "typical_p": full(0.7)}}[cut]
    return dict(kw, temperature=full(0.7), do_sample=torch.ones(rows, device="cuda", dtype=torch.uint8),
                seeds=torch.arange(rows, device="cuda"), steps=full(3, torch.int32))


CUTS = ["none", "top_p", "flat_p", "top_k", "both", "typical", "all"]


def _same(a, b):
    assert torch.equal(a[0], b[0]) and torch.equal(a[1].view(torch.int32), b[1].view(torch.int32))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("cut", ["top_p", "top_k"])
def test_negative_zeros_below_a_maximum_of_eight(dtype, cut):
    """The list reaches to 8 below the maximum, here to 0: an entry of -0 is below that and cannot be kept in place of larger ones."""
    from tgi_b200.ops import cuda as K

    K.load()
    x = torch.full((64, 1000), -20.0, device="cuda")
    x[:, 100:300] = -0.0
    x[:, 7] = 8.0
    one = torch.ones(64, device="cuda")
    kw = {"top_p": {"top_p": one * 0.5}, "top_k": {"top_k": one.int()}}[cut]
    ids, lps = K.fused_sample(x.to(dtype), do_sample=one.to(torch.uint8), seeds=torch.arange(64, device="cuda"), steps=one.int(), **kw)
    assert (ids == 7).all() and (lps == 0).all()


@pytest.mark.parametrize("vocab", [32003, 128256])
@pytest.mark.parametrize("cut", CUTS)
def test_a_row_alone_and_in_batches(vocab, cut):
    """1024 threads a row and 512, and rows that start on 16 bytes or not."""
    from tgi_b200.ops import cuda as K

    K.load()
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n = sms + 1
    g = torch.Generator(device="cuda").manual_seed(vocab)
    x = (torch.randn(n, vocab, device="cuda", generator=g) * 2.5).to(torch.bfloat16)
    pen = torch.full((n,), 1.2, device="cuda")
    history = torch.randint(0, vocab, (n, 700), device="cuda", generator=g)
    kw = _params(n, cut)
    many = K.fused_sample(x, history=history, repetition_penalty=pen, **kw)
    part = lambda a, b: K.fused_sample(x[a:b].clone(), history=history[a:b], repetition_penalty=pen[a:b],
                                       **{k: v[a:b] for k, v in kw.items()})
    _same(part(0, sms), [t[:sms] for t in many])
    for i in range(0, sms, 37):
        _same(part(i, i + 1), [t[i:i + 1] for t in many])


@pytest.mark.parametrize("rows", [2, 200])
@pytest.mark.parametrize("cut", CUTS)
def test_order_of_the_history(rows, cut):
    from tgi_b200.ops import cuda as K

    K.load()
    g = torch.Generator(device="cuda").manual_seed(rows)
    x = torch.randn(rows, 50257, device="cuda", generator=g) * 2.5
    pen = torch.full((rows,), 1.3, device="cuda")
    history = torch.randint(0, 50257, (rows, 1500), device="cuda", generator=g)
    kw = _params(rows, cut)
    first = K.fused_sample(x, history=history, repetition_penalty=pen, **kw)
    for _ in range(4):
        history = history[:, torch.randperm(1500, device="cuda", generator=g)]
        _same(K.fused_sample(x, history=history, repetition_penalty=pen, **kw), first)


@pytest.mark.parametrize("rows", [3, 150])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("ids", [2048, 2049, 3072, 3073, 6000])
@pytest.mark.parametrize("cut", ["none", "top_p", "both", "typical"])
def test_long_histories(rows, dtype, ids, cut):
    """Against a penalised copy of the scores."""
    from tgi_b200.ops import cuda as K

    K.load()
    V = 32003
    g = torch.Generator(device="cuda").manual_seed(ids)
    x = (torch.randn(rows, V, device="cuda", generator=g) * 2).to(dtype)
    history = torch.rand(rows, V, device="cuda", generator=g).argsort(1)[:, :ids]
    pen = torch.tensor([1.3, 0.8, 1.0], device="cuda").repeat(rows)[:rows]
    kw = _params(rows, cut)
    _same(K.fused_sample(x, history=history, repetition_penalty=pen, **kw), K.fused_sample(K.penalties(x, history, pen, None), **kw))


@pytest.mark.parametrize("vocab", [5, 1000, 4099])
@pytest.mark.parametrize("cut", CUTS)
def test_nan_among_penalised_entries(vocab, cut):
    """NaN has one place in the order (under every number that is not negative), whichever way an entry is met."""
    from tgi_b200.ops import cuda as K

    K.load()
    g = torch.Generator(device="cuda").manual_seed(vocab)
    x = torch.randn(12, vocab, device="cuda", generator=g) * 3
    x[:, torch.randperm(vocab, device="cuda", generator=g)[:2]] = float("nan")
    x[3] = float("nan")
    x[4, 0] = float("inf")
    kw = _params(12, cut)
    if "top_k" in kw:
        kw["top_k"] = torch.tensor([1, 2, 3, 4], device="cuda", dtype=torch.int32).repeat(3)
    history = torch.randint(0, vocab, (12, 40), device="cuda", generator=g)
    history[:, :2] = x[0].isnan().nonzero()[:2, 0]
    pen = torch.tensor([1.2, 0.7, 1.0], device="cuda").repeat(4)
    got, want = (K.fused_sample(x, history=history, repetition_penalty=pen, **kw), K.fused_sample(K.penalties(x, history, pen, None), **kw))
    assert torch.equal(got[0], want[0]) and torch.equal(got[1].nan_to_num(7e7), want[1].nan_to_num(7e7))
