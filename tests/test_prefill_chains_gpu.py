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
