"""Shares of the persistent GEMM (``ops/csrc/gemm_sm100.cu``): whole tiles in rounds, equal shares with cut tiles, and K splits, with
even and uneven rounds, ragged edges and few CTAs, in both tile shapes and on CTA pairs.

Tolerance: one rounding to bf16 (2^-8 of the value at most) and fp32 sums (2^-24 per addition, at most 2^14 of them, of the
products' magnitudes)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M", [40, 128, 129, 300])
@pytest.mark.parametrize("N,Kd,ctas", [(1832, 192, 2), (1832, 192, 3), (2048, 320, 6), (1280, 12800, 4), (1288, 12800, 8), (520, 4096, 8)])
@pytest.mark.parametrize("pairs", [True, False])
def test_shares(M, N, Kd, ctas, pairs):
    from tgi_b200.ops import cuda as K

    dev = torch.device("cuda", 0)
    g = torch.Generator(device="cuda").manual_seed(N + M)
    x = torch.randn(M, Kd, device=dev, generator=g).to(torch.bfloat16)
    w = (torch.randn(N, Kd, device=dev, generator=g) * 0.05).to(torch.bfloat16)
    bias = torch.randn(N, device=dev, generator=g).to(torch.bfloat16)
    lib = K.load()
    K.set_gemm_pairs(pairs)
    lib.tgi_gemm_set_pair_min_tiles(1)
    try:
        got = K.gemm_bf16(x, w, bias, max_ctas=ctas)
        torch.cuda.synchronize()
    finally:
        K.set_gemm_pairs(True)
        lib.tgi_gemm_set_pair_min_tiles(32)
    assert K.check_status(dev) == 0, "a kernel wait timed out"
    xd, wd = x.double(), w.double()
    want = xd @ wd.t() + bias.double()
    assert ((got.double() - want).abs() <= want.abs() * 2 ** -8 + (xd.abs() @ wd.abs().t() + 1) * 2 ** -10).all()
