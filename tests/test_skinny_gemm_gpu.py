"""GEMMs of a few tokens (``ops/csrc/gemm_skinny_sm100.cu``): edges of blocks, units, walks and token tiles in the three weight
formats against 64-bit products.

Tolerance: the result is rounded to bf16 once (7 stored bits: half a unit is at most 2^-8 of the value) after fp32 sums,
whose error is below 2^-16 of the sum of the products' magnitudes for the depths used here (2^-24 per addition, fewer than
2^8 additions in a chain)."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def dev():
    return torch.device("cuda", 0)


def _check(got, x, w, bias=None):
    from tgi_b200.ops import cuda as K

    torch.cuda.synchronize()
    assert K.check_status(dev()) == 0, "a kernel wait timed out"
    want = x @ w.t()
    if bias is not None:
        want = want + bias.double()
    bound = want.abs() * 2 ** -8 + (x.abs() @ w.abs().t() + 1) * 2 ** -16
    assert ((got.double() - want).abs() <= bound).all()


TOKENS = [1, 8, 9, 16, 17, 24, 25, 32]


@pytest.mark.parametrize("M", TOKENS)
@pytest.mark.parametrize("N,Kd,ctas", [(8, 64, None), (40, 576, None), (200, 4096, 1), (1000, 1024, 3), (4096, 512, None)])
def test_bf16(M, N, Kd, ctas):
    from tgi_b200.ops import cuda as K

    g = torch.Generator(device="cuda").manual_seed(M + N)
    wide = torch.randn(M, Kd + 64, device=dev(), generator=g).to(torch.bfloat16)
    w = (torch.randn(N, Kd, device=dev(), generator=g) * 0.05).to(torch.bfloat16)
    bias = torch.randn(N, device=dev(), generator=g).to(torch.bfloat16)
    x = wide[:, :Kd].contiguous()
    _check(K.gemm_bf16(x, w, bias, max_ctas=ctas), x.double(), w.double(), bias)
    x = wide[:, 16:16 + Kd]                      # read in place from the wider matrix
    _check(K.gemm_bf16(x, w, max_ctas=ctas), x.double(), w.double())


@pytest.mark.parametrize("M", [1, 7, 8])
@pytest.mark.parametrize("N,Kd,ctas", [(8, 128, None), (200, 1152, None), (1000, 2048, 3), (4096, 1024, None)])
def test_fp8(M, N, Kd, ctas):
    from tgi_b200.ops import cuda as K

    g = torch.Generator(device="cuda").manual_seed(M + N)
    xq, xs = K.fp8_quant_act(torch.randn(M, Kd, device=dev(), generator=g).to(torch.bfloat16))
    wq = (torch.randn(N, Kd, device=dev(), generator=g) * 60).clamp(-440, 440).to(torch.float8_e4m3fn)
    ws = torch.exp2(torch.randint(-12, -6, ((N + 127) // 128, Kd // 128), device=dev(), generator=g).float())
    x = (xq.double().view(M, -1, 128) * xs.double()[:, :, None]).view(M, Kd)
    w = (wq.double().view(N, -1, 128) * ws.double().repeat_interleave(128, 0)[:N, :, None]).view(N, Kd)
    _check(K.gemm_fp8_block(xq, xs, wq, ws, max_ctas=ctas), x, w)


@pytest.mark.parametrize("M", TOKENS)
@pytest.mark.parametrize("N,Kd,group,zero", [(8, 256, 128, True), (200, 2304, 128, True), (1000, 2048, 256, True),
                                             (4096, 512, 128, False), (264, 1024, 1024, True)])
def test_int4(M, N, Kd, group, zero):
    from tgi_b200.ops import cuda as K

    g = torch.Generator(device="cuda").manual_seed(M + N)
    x = torch.randn(M, Kd, device=dev(), generator=g).to(torch.bfloat16)
    wq = torch.randint(0, 256, (N, Kd // 2), device=dev(), dtype=torch.uint8, generator=g)
    scale = (torch.rand(Kd // group, N, device=dev(), generator=g) * 0.02 + 0.002).to(torch.float16)
    zp = torch.randint(0, 17, (Kd // group, N), device=dev(), generator=g).to(torch.float16) if zero else None
    bias = torch.randn(N, device=dev(), generator=g).to(torch.bfloat16)
    q = torch.stack([wq & 15, wq >> 4], -1).view(N, Kd // group, group).double()
    z = zp.t().double()[:, :, None] if zero else 8.0
    w = ((q - z) * scale.t().double()[:, :, None]).view(N, Kd)
    got = K.gemm_wq(x, wq, scale, zp, group, 4, bias)
    # the sums are of (128 + q) x with 128 + z times the tokens' sum taken off: products up to 144 instead of 16 scales
    torch.cuda.synchronize()
    assert K.check_status(dev()) == 0, "a kernel wait timed out"
    want = x.double() @ w.t() + bias.double()
    mag = x.double().abs() @ (144 * scale.double().abs().repeat_interleave(group, 0))
    assert ((got.double() - want).abs() <= want.abs() * 2 ** -8 + (mag + 1) * 2 ** -16).all()


def test_full_ring_gives_the_same_result_every_time():
    """32 tokens keep the consumers busier than the weights' copies: a stage given back before its last shared load has
    returned shows as a result that changes from call to call."""
    from tgi_b200.ops import cuda as K

    g = torch.Generator(device="cuda").manual_seed(0)
    x = torch.randn(32, 14336, device=dev(), generator=g).to(torch.bfloat16)
    w = (torch.randn(4096, 14336, device=dev(), generator=g) * 0.02).to(torch.bfloat16)
    first = K.gemm_bf16(x, w)
    _check(first, x.double(), w.double())
    for _ in range(20):
        assert torch.equal(K.gemm_bf16(x, w), first)


@pytest.mark.parametrize("fmt,M", [("bf16", 5), ("fp8", 5), ("int4", 5), ("bf16", 40), ("fp8", 40), ("bf16", 200), ("fp8", 200)])
def test_settled_weights_in_a_captured_step(fmt, M):
    """Weights fetched while the kernel ahead still runs: a captured chain of norms and products gives, replay after replay, what the
    same calls give in plain stream order; few tokens and the persistent GEMM's tile shapes."""
    from tgi_b200.ops import cuda as K

    H, L = 2048, 6
    g = torch.Generator(device="cuda").manual_seed(3)
    norm = torch.ones(H, device=dev(), dtype=torch.bfloat16)
    x = torch.randn(M, H, device=dev(), generator=g).to(torch.bfloat16)
    ws = [torch.randn(H, H, device=dev(), generator=g) * 0.02 for _ in range(L)]
    if fmt == "fp8":
        ws = [((w * 2000).clamp(-440, 440).to(torch.float8_e4m3fn), torch.full((H // 128, H // 128), 2.0 ** -11, device=dev()))
              for w in ws]
    elif fmt == "int4":
        ws = [(torch.randint(0, 256, (H, H // 2), device=dev(), dtype=torch.uint8, generator=g),
               torch.full((H // 128, H), 0.004, device=dev(), dtype=torch.float16)) for _ in ws]
    else:
        ws = [w.to(torch.bfloat16) for w in ws]

    def step(settled):
        y = x
        for w in ws:
            if fmt == "fp8":
                q, s, _ = K.rms_norm_quant(y, None, norm, 1e-5)
                y = K.gemm_fp8_block(q, s, w[0], w[1], settled=settled)
            else:
                h, _ = K.rms_norm(y, None, norm, 1e-5)
                y = K.gemm_wq(h, w[0], w[1], None, 128, 4, settled=settled) if fmt == "int4" else K.gemm_bf16(h, w, settled=settled)
        return y

    want = step(False)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = step(True)
    for _ in range(20):
        got.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert K.check_status(dev()) == 0 and torch.equal(got, want)


@pytest.mark.parametrize("fmt", ["bf16", "fp8", "int4"])
def test_equal_tokens_give_equal_rows(fmt):
    """Wherever a token stands in its batch and however many there are, up to the largest batches of these kernels."""
    from tgi_b200.ops import cuda as K

    g = torch.Generator(device="cuda").manual_seed(1)
    one = torch.randn(1, 2048, device=dev(), generator=g).to(torch.bfloat16)
    wq = torch.randint(0, 256, (520, 1024), device=dev(), dtype=torch.uint8, generator=g)
    scale = (torch.rand(16, 520, device=dev(), generator=g) * 0.02 + 0.002).to(torch.float16)
    w = (torch.randn(520, 2048, device=dev(), generator=g) * 0.05).to(torch.bfloat16)
    first = None
    for M in range(1, 9 if fmt == "fp8" else 33):
        x = one.expand(M, -1).contiguous()
        if fmt == "int4":
            y = K.gemm_wq(x, wq, scale, None, 128, 4)
        elif fmt == "bf16":
            y = K.gemm_bf16(x, w)
        else:
            y = K.gemm_fp8_block(*K.fp8_quant_act(x), w.to(torch.float8_e4m3fn), torch.ones(5, 16, device=dev()))
        first = y if first is None else first
        assert torch.equal(y, first.expand(M, -1)), M


@pytest.mark.parametrize("fmt", ["bf16", "fp8"])
@pytest.mark.parametrize("M,N,Kd", [(200, 8192, 8192), (300, 4096, 8192)])
def test_settled_weights_on_pairs(fmt, M, N, Kd):
    """At least 32 tiles of 256 x 256 run on CTA pairs: both CTAs' weights go to the leader's barriers ahead of the wait, with many more K
    blocks to a pair than stages."""
    from tgi_b200.ops import cuda as K

    g = torch.Generator(device="cuda").manual_seed(M)
    norm = torch.ones(Kd, device=dev(), dtype=torch.bfloat16)
    xs = [torch.randn(M, Kd, device=dev(), generator=g).to(torch.bfloat16) for _ in range(3)]
    w = torch.randn(N, Kd, device=dev(), generator=g) * 0.02
    w = ((w * 2000).clamp(-440, 440).to(torch.float8_e4m3fn), torch.full((N // 128, Kd // 128), 2.0 ** -11, device=dev())) \
        if fmt == "fp8" else w.to(torch.bfloat16)

    def step(settled):
        if fmt == "fp8":
            return [K.gemm_fp8_block(*K.rms_norm_quant(x, None, norm, 1e-5)[:2], *w, settled=settled) for x in xs]
        return [K.gemm_bf16(K.rms_norm(x, None, norm, 1e-5)[0], w, settled=settled) for x in xs]

    want = step(False)
    assert K.load().tgi_gemm_last_grid() % 2 == 0
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = step(True)
    for _ in range(10):
        for y in got:
            y.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert K.check_status(dev()) == 0 and all(torch.equal(a, b) for a, b in zip(got, want))


@pytest.mark.parametrize("batch", [3, 40, 200])
@pytest.mark.parametrize("pages", [torch.bfloat16, torch.float8_e4m3fn])
def test_settled_weights_behind_decode_attention(batch, pages):
    """A captured chain of decode attention (split and merged for few sequences) and products that fetch their weights meanwhile."""
    from tgi_b200.ops import cuda as K

    heads, kv_heads, L = 16, 4, 1500 if batch < 100 else 200
    g = torch.Generator(device="cuda").manual_seed(batch)
    blocks = (L + 15) // 16
    kc, vc = (torch.randn(batch * blocks, 16, kv_heads, 128, device=dev(), generator=g).to(pages) for _ in range(2))
    table = torch.randperm(batch * blocks, device=dev(), generator=g).int().view(batch, blocks)
    kv = (torch.rand(batch, device=dev(), generator=g) * (L - 1) + 1).int()
    cu = torch.arange(batch + 1, device=dev(), dtype=torch.int32)
    one = torch.ones(kv_heads, device=dev()) if pages != torch.bfloat16 else None
    ws = [(torch.randn(heads * 128, heads * 128, device=dev(), generator=g) * 0.05).to(torch.bfloat16) for _ in range(4)]
    x = torch.randn(batch, heads * 128, device=dev(), generator=g).to(torch.bfloat16)

    def step(settled):
        y = x
        for w in ws:
            o = K.paged_attention(y.view(batch, heads, 128), kc, vc, table, cu, kv, 128 ** -0.5, -1, 0.0, one, one, 1, L)
            y = K.gemm_bf16(o.view(batch, -1), w, settled=settled)
        return y

    want = step(False)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = step(True)
    for _ in range(20):
        got.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert K.check_status(dev()) == 0 and torch.equal(got, want)


def test_fp8_tokens_alone_and_among_others():
    """From 9 tokens on a token's product is the same in every batch up to 128, to the bit; with up to 8 its sums have another order, so
    it is the same but for roundings."""
    from tgi_b200.ops import cuda as K

    g = torch.Generator(device="cuda").manual_seed(5)
    N, Kd = 1024, 4096
    q, s = K.fp8_quant_act(torch.randn(128, Kd, device=dev(), generator=g).to(torch.bfloat16))
    wq = (torch.randn(N, Kd, device=dev(), generator=g) * 60).clamp(-440, 440).to(torch.float8_e4m3fn)
    ws = torch.exp2(torch.randint(-12, -6, (N // 128, Kd // 128), device=dev(), generator=g).float())

    def first(M):
        scales = K.alloc_act_scales(M, Kd // 128, dev())
        scales.copy_(s[:M])
        return K.gemm_fp8_block(q[:M].contiguous(), scales, wq, ws)

    most = first(128)
    for M in (9, 16, 17, 64):
        assert torch.equal(first(M), most[:M]), M
    x = (q.double().view(128, -1, 128) * s.double()[:, :, None]).view(128, Kd)[:8]
    w = (wq.double().view(N, -1, 128) * ws.double().repeat_interleave(128, 0)[:N, :, None]).view(N, Kd)
    for M in (1, 5, 8):
        bound = (x[:M] @ w.t()).abs() * 2 ** -7 + (x[:M].abs() @ w.abs().t()) * 2 ** -15
        assert ((first(M).double() - most[:M].double()).abs() <= bound).all(), M
