"""Performance cases of the serving engine: engine steps as the shard runs them, and the sampling of a step.

A case is one step of ``FlashCausalLM`` on the shapes that this repository's benchmark serves (Llama-3-8B in bf16 and with 4-bit
GPTQ weights, Llama-3-70B in block-scaled fp8 with an fp8 KV cache, Mixtral-8x7B in bf16) with fewer layers, so that a model is
made in about a second and three of them fit the card; all other sizes are the models' own.  Layers are all alike, so the share of
a kernel is that of the whole model except for the head's, which is larger here.

``step``:

* ``decode``: one new token for each of ``batch`` sequences with ``context`` cached tokens on average (half to one and a half of it,
  as requests of different ages have), through the captured decode graphs, from the host's ids to the logits.
* ``prefill``: ``batch`` prompts of ``tokens`` new tokens on average on top of ``context`` cached ones (a shared prefix, or
  the earlier chunks of a long prompt) through ``build_meta`` and ``forward``, to the logits of the prompts' last tokens.
* ``sample``: the sampler of a step over ``batch`` rows of logits with histories of ``context`` tokens.

A sequence's pages lie anywhere in the pool, as they do in a server that has run for a while.
"""
from __future__ import annotations

import math
import zlib

import numpy as np
import torch

from tgi_b200.models.arch import ModelConfig
from tgi_b200.models.decoder import CausalDecoder
from tgi_b200.models.flash_causal_lm import BLOCK_SIZE, FlashCausalLM, FlashCausalLMBatch
from tgi_b200.models.graphs import DEFAULT_BUCKETS, DecodeGraphs
from tgi_b200.ops import cuda as kernels
from tgi_b200.proto import generate_v3 as pb
from tgi_b200.utils import synthetic
from tgi_b200.utils.quantization import DefaultWeightsLoader, Fp8Loader, GPTQLoader
from tgi_b200.utils.tokenizer import ByteTokenizer
from tgi_b200.utils.tokens import NextTokenChooser

FP8 = torch.float8_e4m3fn
KV_SCALE = 0.05         # of the fp8 KV cache, per head
GROUP = 128             # input features per scale of the 4-bit weights
STD = 0.02              # of the weights (see _std for those that write to the residual stream)

# layers that are made, and the models' own sizes
MODELS = {
    "llama8b-bf16": (16, synthetic.llama3_8b_config),
    "llama8b-gptq": (16, synthetic.llama3_8b_config),
    "llama70b-fp8": (8, synthetic.llama3_70b_config),
    "mixtral-bf16": (4, synthetic.mixtral_8x7b_config),
}


def listed():
    return [
        # one user chatting with an idle server: the weights are read for a single row
        {"name": "decode_8b_one", "model": "llama8b-bf16", "step": "decode", "batch": 1, "tokens": 1, "context": 700},
        # a lightly loaded server; 19 sequences run in the graph of 32
        {"name": "decode_8b_few", "model": "llama8b-bf16", "step": "decode", "batch": 19, "tokens": 1, "context": 900},
        # a loaded server at nearly the largest batch of its graphs
        {"name": "decode_8b_many", "model": "llama8b-bf16", "step": "decode", "batch": 201, "tokens": 1, "context": 1100},
        # time to first token of a short question
        {"name": "prompt_8b_short", "model": "llama8b-bf16", "step": "prefill", "batch": 1, "tokens": 77, "context": 0},
        # an 8192-token chunk of a long document, 20k tokens into it
        {"name": "prompt_8b_long", "model": "llama8b-bf16", "step": "prefill", "batch": 1, "tokens": 8192, "context": 20480},
        # the benchmark's headline: full batch of 1024-token prompts in the middle of 512 output tokens
        {"name": "decode_70b_many", "model": "llama70b-fp8", "step": "decode", "batch": 256, "tokens": 1, "context": 1272},
        # the same server with little to do
        {"name": "decode_70b_few", "model": "llama70b-fp8", "step": "decode", "batch": 8, "tokens": 1, "context": 1272},
        # a few prompts that arrived together
        {"name": "prompts_70b", "model": "llama70b-fp8", "step": "prefill", "batch": 3, "tokens": 1100, "context": 0},
        # mixture of experts under a middling load: every expert is read for a few rows
        {"name": "decode_moe", "model": "mixtral-bf16", "step": "decode", "batch": 48, "tokens": 1, "context": 700},
        {"name": "prompts_moe", "model": "mixtral-bf16", "step": "prefill", "batch": 3, "tokens": 683, "context": 0},
        # a 4-bit model on a small deployment
        {"name": "decode_gptq", "model": "llama8b-gptq", "step": "decode", "batch": 12, "tokens": 1, "context": 900},
        # sampled chat at full batch: temperature, top-p and a repetition penalty
        {"name": "sample_nucleus", "model": "llama8b-bf16", "step": "sample", "batch": 256, "tokens": 1, "context": 700,
         "top_k": 0},
    ]


def _spread(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    step = rng.choice(["decode", "decode", "decode", "prefill", "prefill", "sample"])
    if step == "sample":
        return {"model": rng.choice(["llama8b-bf16", "mixtral-bf16"]), "step": step, "batch": _spread(rng, 1, 256), "tokens": 1,
                "context": _spread(rng, 16, 2048), "top_k": rng.choice([0, 0, 20, 50])}
    model = rng.choice(list(MODELS))
    if step == "decode":
        return {"model": model, "step": step, "batch": _spread(rng, 1, 256), "tokens": 1, "context": _spread(rng, 32, 1272)}
    total = _spread(rng, 16, 8192 if model == "llama8b-bf16" else 3300)
    batch = min(rng.choice([1, 1, 2, 3, 5, 8]), total)
    context = rng.choice([0, 0, _spread(rng, 16, 20480 if model == "llama8b-bf16" and batch == 1 else 2048)])
    return {"model": model, "step": step, "batch": batch, "tokens": max(1, total // batch), "context": context}


# ---- sizes -------------------------------------------------------------------------------------------------------------------
def _lengths(mean, n):
    """``n`` lengths from half to one and a half of ``mean``, the same for every seed."""
    return [mean if n == 1 or mean < 2 else max(1, round(mean * (0.5 + (i * 61 % n) / (n - 1)))) for i in range(n)]


def _config(case):
    layers, make = MODELS[case["model"]]
    cfg = make()
    cfg["num_hidden_layers"] = layers
    cfg["max_position_embeddings"] = 32768
    return cfg


def _sequences(case):
    """(new tokens, cached tokens) of every sequence."""
    new = [1] * case["batch"] if case["step"] == "decode" else _lengths(case["tokens"], case["batch"])
    return list(zip(new, _lengths(case["context"], case["batch"])))


def _linears(cfg):
    """(name, output features, input features) of a layer's projections, without routed experts."""
    H, I, D = cfg["hidden_size"], cfg["intermediate_size"], cfg["hidden_size"] // cfg["num_attention_heads"]
    q, kv = cfg["num_attention_heads"] * D, cfg["num_key_value_heads"] * D
    out = [("self_attn.q_proj", q, H), ("self_attn.k_proj", kv, H), ("self_attn.v_proj", kv, H), ("self_attn.o_proj", H, q)]
    if not cfg.get("num_local_experts"):
        out += [("mlp.gate_proj", I, H), ("mlp.up_proj", I, H), ("mlp.down_proj", H, I)]
    return out


def _std(case, name):
    """Blocks write to the residual stream in proportion to one over the whole model's depth, so that no layer takes it over:
    without that, random layers multiply every rounding (16-bit ones from layer to layer, fp8 ones to a third of the logits)."""
    depth = MODELS[case["model"]][1]()["num_hidden_layers"]
    return STD / depth if name.endswith("o_proj") else STD / (2 * depth) if name.endswith(("down_proj", "w2")) else STD


# ---- inputs, from the seed alone -------------------------------------------------------------------------------------------------
def _random(seed, name, shape, std=1.0):
    g = torch.Generator(device="cuda").manual_seed((zlib.crc32(name.encode()) << 20) + seed)
    return torch.randn(shape, generator=g, device="cuda") * std


def _fp8_blocks(w):
    """e4m3 values and the fp32 scale of each 128 x 128 block."""
    n, k = w.shape
    blocks = w.view(n // 128, 128, k // 128, 128)
    scale = blocks.abs().amax(dim=(1, 3)).clamp_min(1e-12) / 448.0
    return (blocks / scale[:, None, :, None]).view(n, k).to(FP8), scale


def _gptq(w):
    """4-bit values ``[K, N]``, zero points and scales ``[K / group, N]`` (scales exact in bf16 and fp16)."""
    wt = w.t().reshape(-1, GROUP, w.shape[0])
    lo, hi = wt.amin(1).clamp_max(0), wt.amax(1).clamp_min(0)
    scale = ((hi - lo) / 15).clamp_min(1e-5).to(torch.bfloat16).float()
    zero = (-lo / scale).round().clamp(1, 15)
    q = (wt / scale[:, None] + zero[:, None]).round().clamp(0, 15)
    return q.view(w.shape[1], w.shape[0]).to(torch.int32), zero.to(torch.int32), scale


def _pack(v, dim):
    """Eight 4-bit values along ``dim`` in an int32, the first in the lowest bits."""
    v = v.unflatten(dim, (-1, 8))
    shift = torch.arange(0, 32, 4, device=v.device, dtype=torch.int32).view([8 if d == dim + 1 else 1 for d in range(v.dim())])
    return (v << shift).sum(dim + 1, dtype=torch.int64).to(torch.int32)


def _linear_weights(case, seed, name, n, k):
    """A projection as its checkpoint stores it."""
    w = _random(seed, name, (n, k), _std(case, name)).to(torch.bfloat16)
    if case["model"] == "llama70b-fp8":
        q, scale = _fp8_blocks(w.float())
        return {name + ".weight": q, name + ".weight_scale_inv": scale}
    if case["model"] == "llama8b-gptq":
        q, zero, scale = _gptq(w.float())
        return {name + ".qweight": _pack(q, 0), name + ".qzeros": _pack(zero - 1, 1), name + ".scales": scale.to(torch.float16),
                name + ".g_idx": torch.arange(k, device="cuda", dtype=torch.int32) // GROUP}
    return {name + ".weight": w}


def _linear_exact(case, seed, name, n, k):
    """The same projection in 64 bits."""
    w = _random(seed, name, (n, k), _std(case, name)).to(torch.bfloat16)
    if case["model"] == "llama70b-fp8":
        q, scale = _fp8_blocks(w.float())
        return (q.double().view(n // 128, 128, k // 128, 128) * scale.double()[:, None, :, None]).view(n, k)
    if case["model"] == "llama8b-gptq":
        q, zero, scale = _gptq(w.float())
        return ((q.view(-1, GROUP, n) - zero[:, None]).double() * scale.double()[:, None]).view(k, n).t().contiguous()
    return w.double()


def _directions(cfg, seed):
    """Unit vectors that the experts answer to.  Trained routers mostly follow the token and are seldom undecided; here the
    embedding of a token holds the directions of its two experts."""
    d = _random(seed, "directions", (cfg["num_local_experts"], cfg["hidden_size"]))
    return d / d.norm(dim=1, keepdim=True)


def _embedding(case, cfg, seed):
    V, H = cfg["vocab_size"], cfg["hidden_size"]
    if not cfg.get("num_local_experts"):
        return _random(seed, "embed", (V, H)).to(torch.bfloat16)
    e, d = cfg["num_local_experts"], _directions(cfg, seed)
    order = _random(seed, "experts", (V, e)).argsort(dim=1)
    return (_random(seed, "embed", (V, H)) + 12 * d[order[:, 0]] + 8 * d[order[:, 1]]).to(torch.bfloat16)


def _router(cfg, seed, layer):
    perm = _random(seed, f"router.{layer}", (cfg["num_local_experts"],)).argsort()
    return (0.5 * _directions(cfg, seed)[perm]).to(torch.bfloat16)


def _expert_names(layer, e):
    p = f"model.layers.{layer}.block_sparse_moe.experts.{e}"
    return p + ".w1", p + ".w3", p + ".w2"


def _checkpoint(case, cfg, seed):
    H, I = cfg["hidden_size"], cfg["intermediate_size"]
    one = torch.ones(H, dtype=torch.bfloat16, device="cuda")
    sd = {"model.embed_tokens.weight": _embedding(case, cfg, seed), "model.norm.weight": one,
          "lm_head.weight": _random(seed, "lm_head", (cfg["vocab_size"], H), STD).to(torch.bfloat16)}
    for i in range(cfg["num_hidden_layers"]):
        p = f"model.layers.{i}."
        sd[p + "input_layernorm.weight"] = sd[p + "post_attention_layernorm.weight"] = one
        for name, n, k in _linears(cfg):
            sd.update(_linear_weights(case, seed, p + name, n, k))
        if cfg.get("num_local_experts"):
            sd[p + "block_sparse_moe.gate.weight"] = _router(cfg, seed, i)
            for e in range(cfg["num_local_experts"]):
                for name, (n, k) in zip(_expert_names(i, e), ((I, H), (I, H), (H, I))):
                    sd[name + ".weight"] = _random(seed, name, (n, k), _std(case, name)).to(torch.bfloat16)
    return sd


def _pages(case, cfg, seed, layer, blocks):
    """Keys and values of a layer's pool of pages: what the earlier steps have left there (normed rows times weights)."""
    shape = (blocks, BLOCK_SIZE, cfg["num_key_value_heads"], cfg["hidden_size"] // cfg["num_attention_heads"])
    fp8 = case["model"] == "llama70b-fp8"
    std = STD * math.sqrt(cfg["hidden_size"])
    return [_random(seed, f"{kind}.{layer}", shape, std / (KV_SCALE if fp8 else 1)).to(FP8 if fp8 else torch.bfloat16)
            for kind in ("keys", "values")]


def _placement(case, seed):
    """(ids of every sequence up to its last token of this step, its blocks, blocks in the pool)."""
    rng = np.random.default_rng(seed)
    vocab = MODELS[case["model"]][1]()["vocab_size"]
    seqs = _sequences(case)
    ids = [rng.integers(3, vocab, size=new + old).tolist() for new, old in seqs]
    need = [math.ceil((new + old + 16) / BLOCK_SIZE) for new, old in seqs]
    order = (1 + rng.permutation(sum(need))).tolist()            # block 0 is the health probe's
    at = np.cumsum([0] + need)
    return ids, [order[a:b] for a, b in zip(at[:-1], at[1:])], 1 + sum(need)


def _logits(case, seed):
    """Rows as language models give them: a bulk, and a few candidates that stand out from it."""
    vocab, n = MODELS[case["model"]][1]()["vocab_size"], case["batch"]
    x = _random(seed, "bulk", (n, vocab), 2.0)
    top = torch.randint(0, vocab, (n, 64), device="cuda", generator=torch.Generator(device="cuda").manual_seed(seed + 1))
    x.scatter_add_(1, top, 6 + 2 * _random(seed, "peaks", (n, 64)).abs())
    return x.to(torch.bfloat16)


# ---- the cases -----------------------------------------------------------------------------------------------------------------
def _parameters(case, i):
    r = pb.Request(id=i, inputs="")
    sampled = case["step"] == "sample"
    r.parameters.temperature = 0.7 if sampled else 1.0
    r.parameters.top_p = 0.9 if sampled else 1.0
    r.parameters.top_k = case["top_k"] if sampled else 0
    r.parameters.repetition_penalty = 1.1 if sampled else 1.0
    r.parameters.typical_p = 1.0
    r.parameters.do_sample = sampled
    r.parameters.seed = 1000 + i
    r.stopping_parameters.max_new_tokens = 16
    r.stopping_parameters.ignore_eos_token = True
    return r


def prepare(case, seed):
    dev = torch.device("cuda", torch.cuda.current_device())
    if case["step"] == "sample":
        chooser = NextTokenChooser.from_pb([_parameters(case, i).parameters for i in range(case["batch"])], dev)
        lens = _lengths(case["context"], case["batch"])
        rng = np.random.default_rng(seed)
        history = np.zeros((case["batch"], max(lens)), dtype=np.int64)
        vocab = MODELS[case["model"]][1]()["vocab_size"]
        for i, n in enumerate(lens):
            history[i, :n] = rng.integers(3, vocab, size=n)
        return {"case": case, "chooser": chooser, "logits": _logits(case, seed), "history": torch.from_numpy(history).to(dev)}
    cfg = _config(case)
    weights = synthetic.DictWeights(_checkpoint(case, cfg, seed), dev, torch.bfloat16)
    weights.weights_loader = {"llama70b-fp8": lambda: Fp8Loader(weight_block_size=[128, 128]),
                              "llama8b-gptq": lambda: GPTQLoader(4, GROUP, False, "gptq")}.get(case["model"], DefaultWeightsLoader)()
    fp8 = case["model"] == "llama70b-fp8"
    model = CausalDecoder(ModelConfig(cfg), weights)
    del weights
    if fp8:
        for layer in model.layers:
            layer.attn.k_scale = torch.full((cfg["num_key_value_heads"],), KV_SCALE, device=dev)
            layer.attn.v_scale = torch.full((cfg["num_key_value_heads"],), KV_SCALE, device=dev)
    runner = FlashCausalLM(model, ByteTokenizer(cfg["vocab_size"]), torch.bfloat16, dev, kv_cache_dtype=FP8 if fp8 else torch.bfloat16)
    ids, blocks, pool = _placement(case, seed)
    runner.init_kv_cache(pool)
    for i, (k, v) in enumerate(runner.kv_cache):
        for page, value in zip((k, v), _pages(case, cfg, seed, i, pool)):
            page.copy_(value)
    request = pb.Batch(id=0, size=case["batch"])
    for i, b in enumerate(blocks):
        r = _parameters(case, i)
        r.blocks.extend(b)
        request.requests.append(r)
    batch = FlashCausalLMBatch.from_tokenized(request, ids, runner.tokenizer, torch.bfloat16, dev)
    for s, (new, old) in zip(batch.seqs, _sequences(case)):
        s.cache_len, s.prefilling = old, case["step"] == "prefill"
    state = {"case": case, "runner": runner, "batch": batch, "counts": batch.plan_step()}
    if case["step"] == "decode":
        longest = max(len(b) for b in blocks) * BLOCK_SIZE
        runner.graphs = DecodeGraphs(runner, max(4096, longest), buckets=[min(b for b in DEFAULT_BUCKETS if b >= case["batch"])])
        with torch.no_grad():
            runner.graphs.capture_all()
    if kernels.check_status(dev) != 0:
        raise RuntimeError("a kernel's wait ran out")
    return state


@torch.no_grad()
def run(state):
    case = state["case"]
    if case["step"] == "sample":
        chooser = state["chooser"]
        chooser.steps = [5] * case["batch"]          # the same draw in every pass
        ids, logprobs = chooser(state["history"], state["logits"], need_logprobs=False)[:2]
        return {"ids": ids, "logprobs": logprobs}
    runner, batch, counts = state["runner"], state["batch"], state["counts"]
    if case["step"] == "decode":
        logits, _ = runner.graphs.run(batch, counts)
    else:
        meta, _ = runner.build_meta(batch, counts)
        logits = runner.forward(meta)
    keys, values = runner.kv_cache[-1]
    return {"logits": logits, "keys": keys, "values": values}


def work(case):
    cfg = _config(case)
    H, I, V, L = cfg["hidden_size"], cfg["intermediate_size"], cfg["vocab_size"], cfg["num_hidden_layers"]
    if case["step"] == "sample":
        return {"bytes": case["batch"] * (2 * V + 12) + 8 * sum(_lengths(case["context"], case["batch"])), "flops": 0}
    seqs = _sequences(case)
    heads, kv, D = cfg["num_attention_heads"], cfg["num_key_value_heads"], H // cfg["num_attention_heads"]
    T, B = sum(n for n, _ in seqs), len(seqs)
    per_weight = {"llama70b-fp8": 1 + 4 / 128 ** 2, "llama8b-gptq": 0.5 + 2.5 / GROUP}.get(case["model"], 2)
    per_key = 1 if case["model"] == "llama70b-fp8" else 2
    dense = sum(n * k for _, n, k in _linears(cfg))
    weights, products = dense * per_weight, 2 * dense * T
    if cfg.get("num_local_experts"):
        e, top = cfg["num_local_experts"], cfg["num_experts_per_tok"]
        touched = e * (1 - (1 - top / e) ** T)             # expected, with experts chosen evenly
        weights += 2 * (touched * 3 * I * H + e * H)
        products += 2 * T * (top * 3 * I * H + e * H)
    pairs = sum(n * old + n * (n + 1) // 2 for n, old in seqs)
    cached = sum(n + old for n, old in seqs) * 2 * kv * D * per_key
    return {"bytes": L * (weights + cached) + 2 * (V * H + T * H + B * V),
            "flops": L * (products + 4 * pairs * heads * D) + 2 * B * V * H}


def tolerance(case):
    """Measured: the same steps with decode attention, prefill attention and products in their other implementations (sums in
    another order) differ by 0.004 to 0.005 in bf16 (0.002 of Mixtral's shape) and 0.005 to 0.010 in fp8, whose activations are
    quantised anew for every product: one that a sum in another order brings over a rounding boundary moves by a sixteenth."""
    if case["step"] == "sample":
        return {"rel": 1e-4, "max": 1e-3, "differ": 0.004}
    if case["model"] == "llama70b-fp8":
        return {"rel": 0.03, "max": 0.2}
    return {"rel": 0.01, "max": 0.04} if case["model"] == "mixtral-bf16" else {"rel": 0.02, "max": 0.08}


# ---- the same step in 64 bits --------------------------------------------------------------------------------------------------------
def _norm(x, eps):
    return x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + eps)


def _attend(q, k, v, old):
    """Causal attention of ``q[T, H, D]`` (positions from ``old``) over ``k, v[old + T, Hkv, D]``."""
    T, heads, D = q.shape
    group, out = heads // k.shape[1], torch.empty_like(q)
    for h in range(k.shape[1]):
        for a in range(0, T, 1024):
            b = min(T, a + 1024)
            s = torch.einsum("tgd,sd->gts", q[a:b, h * group:(h + 1) * group], k[:old + b, h]) / math.sqrt(D)
            late = torch.arange(old + b, device=q.device)[None] > torch.arange(old + a, old + b, device=q.device)[:, None]
            out[a:b, h * group:(h + 1) * group] = torch.einsum("gts,sd->tgd", s.masked_fill_(late, -math.inf).softmax(-1), v[:old + b, h])
    return out


@torch.no_grad()
def exact(case, seed):
    if case["step"] == "sample":
        return None          # what is drawn has no such value
    cfg = _config(case)
    H, I, eps, theta = cfg["hidden_size"], cfg["intermediate_size"], cfg["rms_norm_eps"], cfg["rope_theta"]
    heads, kv, D = cfg["num_attention_heads"], cfg["num_key_value_heads"], H // cfg["num_attention_heads"]
    unit = KV_SCALE if case["model"] == "llama70b-fp8" else 1.0
    seqs = _sequences(case)
    ids, blocks, pool = _placement(case, seed)
    step_ids = torch.tensor([t for s, (n, old) in zip(ids, seqs) for t in s[old:]], device="cuda")
    pos = torch.tensor([p for n, old in seqs for p in range(old, old + n)], device="cuda")
    inv = 1.0 / theta ** (torch.arange(0, D, 2, device="cuda", dtype=torch.float64) / D)
    angle = pos.double()[:, None] * inv
    cos, sin = angle.cos()[:, None], angle.sin()[:, None]

    def rotate(x):
        a, b = x[..., :D // 2], x[..., D // 2:]
        return torch.cat([a * cos - b * sin, b * cos + a * sin], -1)

    def project(x, name):
        n, k = next((n, k) for m, n, k in _linears(cfg) if name.endswith(m))
        return x @ _linear_exact(case, seed, name, n, k).t()

    rows = np.cumsum([0] + [n for n, _ in seqs])
    slots = [torch.tensor([b[p // BLOCK_SIZE] * BLOCK_SIZE + p % BLOCK_SIZE for p in range(n + old)], device="cuda")
             for b, (n, old) in zip(blocks, seqs)]
    x = _embedding(case, cfg, seed)[step_ids].double()
    T = x.shape[0]
    for i in range(cfg["num_hidden_layers"]):
        p = f"model.layers.{i}."
        h = _norm(x, eps)
        q = rotate(project(h, p + "self_attn.q_proj").view(T, heads, D))
        k = rotate(project(h, p + "self_attn.k_proj").view(T, kv, D))
        v = project(h, p + "self_attn.v_proj").view(T, kv, D)
        keys, values = _pages(case, cfg, seed, i, pool)
        flat = [t.view(-1, kv, D) for t in (keys, values)]
        out = torch.empty_like(q)
        for (a, b), s, (n, old) in zip(zip(rows[:-1], rows[1:]), slots, seqs):
            past = [t.index_select(0, s[:old]).double() * unit for t in flat]
            out[a:b] = _attend(q[a:b], torch.cat([past[0], k[a:b]]), torch.cat([past[1], v[a:b]]), old)
        x = x + project(out.reshape(T, -1), p + "self_attn.o_proj")
        h = _norm(x, eps)
        if cfg.get("num_local_experts"):
            scores = h @ _router(cfg, seed, i).double().t()
            top, which = scores.topk(cfg["num_experts_per_tok"], dim=1)
            weight = top.softmax(-1)
            y = torch.zeros_like(x)
            for e in range(cfg["num_local_experts"]):
                row, slot = (which == e).nonzero(as_tuple=True)
                w1, w3, w2 = (_random(seed, n, s, _std(case, n)).to(torch.bfloat16).double()
                              for n, s in zip(_expert_names(i, e), ((I, H), (I, H), (H, I))))
                y[row] += weight[row, slot, None] * ((torch.nn.functional.silu(h[row] @ w1.t()) * (h[row] @ w3.t())) @ w2.t())
            x = x + y
        else:
            gate = torch.nn.functional.silu(project(h, p + "mlp.gate_proj"))
            x = x + project(gate * project(h, p + "mlp.up_proj"), p + "mlp.down_proj")
    last = torch.from_numpy(rows[1:] - 1).to(x.device)
    head = _random(seed, "lm_head", (cfg["vocab_size"], H), STD).to(torch.bfloat16)
    logits = torch.cat([_norm(x[last], eps) @ w.double().t() for w in head.split(16384)], 1)
    new = torch.cat([s[old:] for s, (n, old) in zip(slots, seqs)])
    keys, values = (t.double() for t in (keys, values))
    keys.view(-1, kv, D)[new], values.view(-1, kv, D)[new] = k / unit, v / unit
    return {"logits": logits, "keys": keys, "values": values}
