"""Prefill attention in two chains of KV tiles (``ops/csrc/attention_prefill_bf16_sm100.cu``): row maxima that outgrow the chains'
reference again and again, shrink, or stay, over one tile, two, an odd and an even number of them.

Tolerance: probabilities are rounded to bf16 (2^-8 of each at most) and so is the result, whose entries are averages of values
below 5: 5 * (2^-8 + 2^-8) with the errors of the sums and of the exponential well below."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,cached", [(1, 100), (100, 0), (128, 128), (130, 255), (200, 900), (257, 1000)])
@pytest.mark.parametrize("trend", ["growing", "shrinking", "flat"])
@pytest.mark.parametrize("softcap", [0.0, 40.0])
def test_row_maxima(n, cached, trend, softcap):
    from tgi_b200.ops import cuda as K, reference as ref

    dev, heads, kv_heads, L = torch.device("cuda", 0), 4, 2, n + cached
    g = torch.Generator(device="cuda").manual_seed(n + cached)
    blocks = (L + 15) // 16
    at = torch.arange(blocks * 16, device=dev).float() / L
    gain = {"growing": 1 + 30 * at, "shrinking": 31 - 30 * at, "flat": torch.ones_like(at)}[trend].view(blocks, 16, 1, 1)
    k = (torch.randn(blocks, 16, kv_heads, 128, device=dev, generator=g) * gain).to(torch.bfloat16)
    v = torch.randn(blocks, 16, kv_heads, 128, device=dev, generator=g).clamp(-5, 5).to(torch.bfloat16)
    q = torch.randn(max(n, 2), heads, 128, device=dev, generator=g).to(torch.bfloat16)      # two tokens: not a decode step
    lens = [n] if n > 1 else [1, 1]
    table = torch.arange(blocks, device=dev, dtype=torch.int32).repeat(len(lens), 1)
    cu = torch.tensor([0] + torch.tensor(lens).cumsum(0).tolist(), device=dev, dtype=torch.int32)
    kv = torch.full((len(lens),), L, device=dev, dtype=torch.int32)
    args = (q, k, v, table, cu, kv, 128 ** -0.5, -1, softcap)
    want = ref.paged_attention(*args, None, None)
    got = K.paged_attention(*args, None, None, max(n, 2), L)
    torch.cuda.synchronize()
    assert K.check_status() == 0
    assert (got.float() - want.float()).abs().max() <= 5 * 2 ** -7


def _relative(got, want):
    """Probabilities and the result are rounded to bf16 (2^-9 on average, at random); a wrong key or order is a matter of 1 / sqrt(keys)."""
    return ((got.double() - want.double()).norm() / want.double().norm()).item()


@pytest.mark.parametrize("n,cached", [(128, 0), (130, 255), (300, 700)])
@pytest.mark.parametrize("what", ["window", "kept", "kept_tiles", "horizon", "sink", "chunk", "all"])
def test_masks_and_sinks(n, cached, what):
    """Kept first tokens come in tiles of their own, so the parity of the window's tiles changes with them."""
    from tgi_b200.ops import cuda as K, reference as ref

    dev, heads, kv_heads, L = torch.device("cuda", 0), 4, 2, n + cached
    g = torch.Generator(device="cuda").manual_seed(n)
    blocks = (L + 15) // 16
    k, v = (torch.randn(blocks + 5, 16, kv_heads, 128, device=dev, generator=g).to(torch.bfloat16) for _ in range(2))
    q = torch.randn(n, heads, 128, device=dev, generator=g).to(torch.bfloat16)
    table = torch.randperm(blocks + 5, device=dev, generator=g)[:blocks].int().view(1, -1)
    cu, kv = torch.tensor([0, n], device=dev, dtype=torch.int32), torch.tensor([L], device=dev, dtype=torch.int32)
    pos = torch.arange(cached, L, device=dev, dtype=torch.int32)
    kw = {"window": {"window": 100}, "kept": {"window": 70, "keep": 4}, "kept_tiles": {"window": 70, "keep": 200},
          "horizon": {"horizon": pos // 50 * 50 + 49}, "sink": {"sink": torch.randn(heads, device=dev, generator=g) * 3},
          "chunk": {"chunk": 96}, "all": {"window": 150, "keep": 130, "softcap": 20.0, "sink": torch.randn(heads, device=dev, generator=g)}}[what]
    want = ref.paged_attention(q, k, v, table, cu, kv, 128 ** -0.5, **kw)
    got = K.paged_attention(q, k, v, table, cu, kv, 128 ** -0.5, max_q=n, max_kv=L, **kw)
    torch.cuda.synchronize()
    assert K.check_status() == 0 and _relative(got, want) < 2 ** -7


@pytest.mark.parametrize("dim", [128, 192])
@pytest.mark.parametrize("lens", [[(1, 0)], [(128, 0), (129, 0)], [(257, 400), (60, 900), (200, 3)]])
@pytest.mark.parametrize("window,gated,sunk", [(-1, False, False), (90, True, False), (-1, True, True), (300, False, True)])
def test_keys_and_values_written_out(dim, lens, window, gated, sunk):
    """192-wide queries and keys share one tile of values and one of probabilities between the chains."""
    from types import SimpleNamespace

    from tgi_b200.ops import cuda as K, reference as ref

    dev, heads = torch.device("cuda", 0), 3
    g = torch.Generator(device="cuda").manual_seed(dim + len(lens))
    T, blocks = sum(n for n, _ in lens), [(n + c + 15) // 16 for n, c in lens]
    R = 16 * sum(blocks)
    kv = torch.randn(R, heads * (dim + 128), device=dev, generator=g).to(torch.bfloat16)
    q = torch.randn(T, heads, dim, device=dev, generator=g).to(torch.bfloat16)
    tables = torch.zeros(len(lens), max(blocks), device=dev, dtype=torch.int32)
    order = torch.randperm(R // 16, device=dev, generator=g).int()
    for i, b in enumerate(blocks):
        tables[i, :b] = order[sum(blocks[:i]):sum(blocks[:i]) + b]
    cu = torch.tensor([0] + torch.tensor([n for n, _ in lens]).cumsum(0).tolist(), device=dev, dtype=torch.int32)
    held = torch.tensor([n + c for n, c in lens], device=dev, dtype=torch.int32)
    gate = torch.randn(T, heads + 5, device=dev, generator=g).to(torch.bfloat16)[:, 2:2 + heads] if gated else None
    sink = torch.randn(heads, device=dev, generator=g) * 2 if sunk else None
    keys = kv[:, :heads * dim].reshape(R // 16, 16, heads, dim).contiguous()
    values = kv[:, heads * dim:].reshape(R // 16, 16, heads, 128).contiguous()
    want = ref.paged_attention(q, keys, values, tables, cu, held, 0.07, window, sink=sink).float()
    if gated:
        want = want * gate.float().sigmoid()[:, :, None]
    out = torch.empty(T, heads, 128, device=dev, dtype=torch.bfloat16)
    K.expanded_attention(q, kv, SimpleNamespace(tables=tables, kv_lens=held), cu, 0.07, window, max(n for n, _ in lens), gate, out, sink)
    torch.cuda.synchronize()
    assert K.check_status() == 0 and _relative(out, want) < 2 ** -7
    flat, truth = out.view(T, -1).double(), want.view(T, -1).double()
    assert ((flat - truth).norm(dim=1) <= 2 ** -6 * truth.norm(dim=1) + 1e-3).all()
