"""Shares of the persistent GEMM (``ops/csrc/gemm_sm100.cu``): whole tiles in rounds, equal shares with cut tiles, and K splits, with
even and uneven rounds, ragged edges and few CTAs, in both tile shapes and on CTA pairs, in bf16 and in both modes of fp8.

Tolerance: one rounding to bf16 (2^-8 of the value at most) and fp32 sums, which the tensor core rounds once per 16 features (2^-23
of the products' magnitudes each, at most 2^10 times); a K block that is missing or met twice is several times that."""
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
    assert ((got.double() - want).abs() <= want.abs() * 2 ** -8 + (xd.abs() @ wd.abs().t() + 1) * 2 ** -13).all()


@pytest.fixture
def small_pairs():
    """Pairs for problems of any size; the fp8 mode comes back as it was."""
    from tgi_b200.ops import cuda as K

    lib = K.load()
    mode = K.fp8_mx()
    lib.tgi_gemm_set_pair_min_tiles(1)
    yield K
    lib.tgi_gemm_set_pair_min_tiles(32)
    K.set_fp8_mx(mode)


def _fp8(K, M, N, Kd, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    q, s = K.fp8_quant_act(torch.randn(M, Kd, device="cuda", generator=g).to(torch.bfloat16))
    w = (torch.randn(N, Kd, device="cuda", generator=g) * 60).clamp(-440, 440).to(torch.float8_e4m3fn)
    ws = torch.exp2(torch.randint(-12, -6, ((N + 127) // 128, Kd // 128), device="cuda", generator=g).float())
    return q, s, w, ws


@pytest.mark.parametrize("M", [40, 128, 129, 200, 300])
@pytest.mark.parametrize("N,Kd,ctas", [(1832, 384, 2), (1832, 384, 3), (2048, 640, 6), (1280, 8576, 8), (1288, 2560, 8), (520, 4096, 8)])
@pytest.mark.parametrize("mx", [True, False])
def test_shares_fp8(small_pairs, M, N, Kd, ctas, mx):
    """One rounding to bf16; the tensor core rounds its fp32 sum once per 32 features (2^-23 each, at most 2^9 of them)."""
    K = small_pairs
    K.set_fp8_mx(mx)
    q, s, w, ws = _fp8(K, M, N, Kd, N + M)
    got = K.gemm_fp8_block(q, s, w, ws, max_ctas=ctas)
    torch.cuda.synchronize()
    assert K.check_status(q.device) == 0, "a kernel wait timed out"
    x = (q.double().view(M, -1, 128) * s.double()[:, :, None]).view(M, Kd)
    wd = (w.double().view(N, -1, 128) * ws.double().repeat_interleave(128, 0)[:N, :, None]).view(N, Kd)
    want = x @ wd.t()
    assert ((got.double() - want).abs() <= want.abs() * 2 ** -8 + (x.abs() @ wd.abs().t()) * 2 ** -14 + 1e-30).all()


@pytest.mark.parametrize("fmt,M,blocks,whole", [
    ("bf16", 200, 88, True), ("bf16", 200, 96, False), ("mx", 200, 52, True), ("mx", 200, 56, False), ("mx", 40, 72, True),
    ("mx", 40, 80, False), ("promotion", 200, 28, True), ("promotion", 200, 36, False), ("promotion", 40, 24, True), ("promotion", 40, 32, False)])
def test_whole_tiles_where_they_cost_less(small_pairs, fmt, M, blocks, whole):
    """One tile more than workers: two rounds of whole tiles take nearly twice an equal share of K blocks."""
    K = small_pairs
    N, grid = (1280, 6) if M > 128 else (2304, 5)
    if fmt == "bf16":
        K.gemm_bf16(torch.zeros(M, 64 * blocks, device="cuda", dtype=torch.bfloat16),
                    torch.zeros(N, 64 * blocks, device="cuda", dtype=torch.bfloat16), max_ctas=8)
    else:
        K.set_fp8_mx(fmt == "mx")
        K.gemm_fp8_block(*_fp8(K, M, N, 128 * blocks, 1), max_ctas=8)
    torch.cuda.synchronize()
    assert K.load().tgi_gemm_last_grid() == (grid if whole else 8)
