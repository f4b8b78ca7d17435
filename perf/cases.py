"""What this framework's speed is measured on: the work of serving, through the public op layer and the engine.

Every case is one pass of a step that a served model takes - attention over the paged cache, latent attention, a gated
delta-net layer's core, a block of routed experts, a dense feed-forward, a whole decoder - at the sizes of the presets in
``vllm_kunlun_b200/config.py``, of ``bench.py`` and of the scripts under ``benchmarks/``.  A step of prompt portions and a step of
decoding are cases of their own, because they are bound by different things.

``listed()``: the fixed cases; ``draw(rng)``: one more of the same ranges; ``prepare(case, seed)``: inputs, weights and what a
serving process keeps between steps; ``run(state)``: one pass; ``work(case)``: the bytes and operations that a pass cannot do
without; ``tolerance(case)``; ``exact(case, seed)``: the same result in plain 64-bit torch.
"""
import math

import torch

DEV = "cuda"
DTYPES = {"bf16": torch.bfloat16, "fp16": torch.float16}
BLOCK = 64                    # tokens of a cache block, as in bench.py and the replay command

# heads and key / value heads (head size 128): Llama-3.1-8B and Qwen3-8B, Qwen3-30B-A3B, the "small" layer-benchmark size
HEADS = [(32, 8), (32, 4), (16, 4)]
# key heads and value heads of a gated delta net (128 each): Qwen3-Next on one GPU and on one of two, the layer benchmark
GDN_HEADS = [(16, 32), (8, 16), (16, 16)]
# width, experts, experts per token, expert width: Qwen3-30B-A3B, the two layer-benchmark sizes
EXPERTS = [(2048, 128, 8, 768), (2048, 32, 4, 768), (4096, 32, 4, 1536)]
# width and feed-forward width: Llama-3.1-8B, Qwen3-8B, the small layer-benchmark size
FEED_FORWARD = [(4096, 14336), (4096, 12288), (2048, 6144)]
# width, feed-forward width, heads, key / value heads, layers, vocabulary: the layer-benchmark sizes, four layers of them
MODELS = [(4096, 12288, 32, 8, 4, 32000), (2048, 6144, 16, 4, 4, 32000)]


# ----------------------------------------------------------------------------- the cases

def listed():
    return [
        # Prefill attention of the headline benchmark: one step takes four 2048-token prompts (8192 tokens a step).
        dict(name="attn_prefill_4x2048", kind="attn", heads=32, kv_heads=8, requests=4, new=2048, context=0, ragged=False,
             window=0, dtype="bf16"),
        # A long prompt: the last 8192-token portion of 32768 tokens, Qwen3-30B-A3B heads.
        dict(name="attn_chunk_8k_of_32k", kind="attn", heads=32, kv_heads=4, requests=1, new=8192, context=24576,
             ragged=False, window=0, dtype="bf16"),
        # Short prompts of uneven lengths in one step, as chat requests arrive.
        dict(name="attn_prefill_ragged", kind="attn", heads=32, kv_heads=8, requests=11, new=371, context=0, ragged=True,
             window=0, dtype="bf16"),
        # Decode attention of the headline benchmark half way through: 16 requests with 3072 tokens each.
        dict(name="attn_decode_16x3072", kind="attn", heads=32, kv_heads=8, requests=16, new=1, context=3071, ragged=False,
             window=0, dtype="bf16"),
        # One interactive request with a short history: the smallest call, where latency and launches count.
        dict(name="attn_decode_1x900", kind="attn", heads=32, kv_heads=8, requests=1, new=1, context=899, ragged=False,
             window=0, dtype="bf16"),
        # Latent attention (DeepSeek-V3 heads of one of eight ranks): prompts in the up-projected form, and decoding.
        dict(name="mla_prefill_4x2048", kind="mla_prefill", heads=16, requests=4, new=2048, context=0, ragged=False,
             dtype="bf16"),
        dict(name="mla_decode_16x4096", kind="mla_decode", heads=16, requests=16, new=1, context=4095, ragged=False,
             dtype="bf16"),
        # Gated delta net (Qwen3-Next): convolution, gates, recurrence and gated norm of one layer, prompts and decoding.
        dict(name="gdn_prefill_4x2048", kind="gdn", k_heads=16, v_heads=32, requests=4, new=2048, ragged=False, carried=False),
        dict(name="gdn_decode_64", kind="gdn", k_heads=16, v_heads=32, requests=64, new=1, ragged=False, carried=True),
        # Routed experts (Qwen3-30B-A3B, fp8 weights with 128 x 128 block scales): a prompt portion, and 16 decoding requests.
        dict(name="moe_prefill_4096", kind="moe", size=0, tokens=4096, fp8=True),
        dict(name="moe_decode_16", kind="moe", size=0, tokens=16, fp8=True),
        # A dense decoder through the engine, prompt tokens in, logits out (8B widths, four layers).
        dict(name="model_prefill_4x2048", kind="model", size=0, requests=4, new=2048, ragged=False),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["attn", "attn_decode", "mla_prefill", "mla_decode", "gdn", "gdn_decode", "moe", "moe_decode", "mlp", "model"])
    ragged = rng.random() < 0.5
    if kind in ("attn", "attn_decode"):
        heads, kv = rng.choice(HEADS)
        c = dict(kind="attn", heads=heads, kv_heads=kv, ragged=ragged, dtype=rng.choice(["bf16", "bf16", "fp16"]),
                 window=rng.choice([0, 0, 0, 1024]))
        if kind == "attn":
            requests = _log(rng, 1, 16)
            new = _log(rng, 24, 8192 // requests)
            context = rng.choice([0, _log(rng, 1, 16384)])
        else:
            requests = _log(rng, 1, 64)
            new, context = 1, _log(rng, 30, min(32767, 131072 // requests))
        return dict(c, requests=requests, new=new, context=context)
    if kind == "mla_prefill":
        requests = _log(rng, 1, 8)
        return dict(kind=kind, heads=rng.choice([16, 32]), requests=requests, new=_log(rng, 24, 8192 // requests), context=0,
                    ragged=ragged, dtype="bf16")
    if kind == "mla_decode":
        requests = _log(rng, 1, 64)
        return dict(kind=kind, heads=rng.choice([16, 16, 32, 128]), requests=requests, new=rng.choice([1, 1, 2]),
                    context=_log(rng, 30, min(16384, 131072 // requests)), ragged=ragged, dtype="bf16")
    if kind in ("gdn", "gdn_decode"):
        k_heads, v_heads = rng.choice(GDN_HEADS)
        if kind == "gdn":
            requests = _log(rng, 1, 8)
            new, carried = _log(rng, 24, min(4096, 8192 // requests)), rng.random() < 0.5
        else:
            requests, new, carried, ragged = _log(rng, 1, 128), 1, True, False
        return dict(kind="gdn", k_heads=k_heads, v_heads=v_heads, requests=requests, new=new, ragged=ragged, carried=carried)
    if kind in ("moe", "moe_decode"):
        return dict(kind="moe", size=rng.randrange(len(EXPERTS)), fp8=rng.random() < 0.6,
                    tokens=_log(rng, 65, 8192) if kind == "moe" else _log(rng, 1, 64))
    if kind == "mlp":
        return dict(kind="mlp", size=rng.randrange(len(FEED_FORWARD)), tokens=_log(rng, 1, 4096), dtype="bf16")
    requests = _log(rng, 1, 8)
    return dict(kind="model", size=rng.randrange(len(MODELS)), requests=requests, new=_log(rng, 24, 8192 // requests),
                ragged=ragged)


# ----------------------------------------------------------------------------- inputs

def _lengths(case):
    """New tokens and earlier tokens of every request; ragged: between a third of the given size and all of it."""
    n, R = case["new"], case["requests"]
    context = case.get("context", 0)
    if not case["ragged"]:
        return [n] * R, [context] * R
    share = [(1 + (5 * i + 3) % 7 / 3) / 3 for i in range(R)]
    return [max(1, int(n * s)) for s in share], [int(context * s) for s in share]


def _starts(lens):
    out = [0]
    for n in lens:
        out.append(out[-1] + n)
    return out


def _gen(seed):
    return torch.Generator(device=DEV).manual_seed(seed)


def _randn(g, *shape, dtype=torch.bfloat16, scale=1.0):
    return (torch.randn(*shape, generator=g, device=DEV) * scale).to(dtype)


def _ints(values):
    return torch.tensor(values, dtype=torch.int32, device=DEV)


def _paged(g, lens):
    """Block tables of requests with these lengths, blocks in random order as a used pool hands them out."""
    need = [-(-n // BLOCK) for n in lens]
    order = torch.randperm(sum(need), generator=g, device=DEV).to(torch.int32)
    table = torch.zeros(len(lens), max(need), dtype=torch.int32, device=DEV)
    at = 0
    for i, n in enumerate(need):
        table[i, :n] = order[at:at + n]
        at += n
    return table, sum(need)


def _fp8_blocks(w):
    """``[E, N, K]`` in e4m3 with a scale per 128 x 128 block (largest magnitude = 448)."""
    E, N, K = w.shape
    b = w.float().view(E, N // 128, 128, K // 128, 128)
    scale = b.abs().amax((2, 4)).clamp_min(1e-12) / 448.0
    return (b / scale[:, :, None, :, None]).view(E, N, K).to(torch.float8_e4m3fn), scale.contiguous()


def _inputs(case, seed):
    """The numbers of a case: plain tensors, made from the seed alone."""
    g = _gen(seed)
    kind = case["kind"]
    if kind in ("attn", "mla_decode"):
        dt = DTYPES[case["dtype"]]
        new, ctx = _lengths(case)
        lens = [a + b for a, b in zip(new, ctx)]
        table, blocks = _paged(g, lens)
        i = dict(new=new, lens=lens, table=table, seq_lens=_ints(lens), qsl=_ints(_starts(new)), T=sum(new))
        if kind == "attn":
            i.update(q=_randn(g, i["T"], case["heads"], 128, dtype=dt), scale=128 ** -0.5,
                     cache=_randn(g, blocks, 2, case["kv_heads"], BLOCK, 128, dtype=dt))
        else:
            i.update(q=_randn(g, i["T"], case["heads"], 576, dtype=dt), cache=_randn(g, blocks, BLOCK, 576, dtype=dt, scale=0.3),
                     scale=192 ** -0.5)
        return i
    if kind == "mla_prefill":
        dt = DTYPES[case["dtype"]]
        new, _ = _lengths(case)
        T, N = sum(new), case["heads"]
        return dict(new=new, T=T, qsl=_ints(_starts(new)), lens=_ints(new), q=_randn(g, T, N, 192, dtype=dt),
                    kv=_randn(g, T, N * 256, dtype=dt), k_pe=_randn(g, T, 64, dtype=dt), scale=192 ** -0.5)
    if kind == "gdn":
        Hk, Hv, R = case["k_heads"], case["v_heads"], case["requests"]
        new, _ = _lengths(case)
        T, C = sum(new), (2 * Hk + Hv) * 128
        states = torch.randn(R, Hv, 128, 128, generator=g, device=DEV) * 0.1
        return dict(new=new, T=T, C=C, cu=_ints(_starts(new)), slots=torch.randperm(R, generator=g, device=DEV).to(torch.int32),
                    init=torch.full((R,), int(case["carried"]), dtype=torch.int32, device=DEV),
                    qkvz=_randn(g, T, C + Hv * 128), ba=_randn(g, T, 2 * Hv), conv_w=_randn(g, C, 4, scale=0.3),
                    conv_state=_randn(g, R, 3, C), states=states, norm_w=(1 + _randn(g, 128, scale=0.1)).to(torch.bfloat16),
                    A_log=torch.rand(Hv, generator=g, device=DEV) * 2 - 1, dt_bias=torch.rand(Hv, generator=g, device=DEV) * 2 - 1)
    if kind == "moe":
        H, E, k, I = EXPERTS[case["size"]]
        i = dict(x=_randn(g, case["tokens"], H), logits=torch.randn(case["tokens"], E, generator=g, device=DEV), k=k,
                 w13_scale=None, w2_scale=None)
        i["w13"], i["w2"] = _randn(g, E, 2 * I, H, scale=0.02), _randn(g, E, H, I, scale=0.02)
        if case["fp8"]:
            i["w13"], i["w13_scale"] = _fp8_blocks(i["w13"])
            i["w2"], i["w2_scale"] = _fp8_blocks(i["w2"])
        return i
    if kind == "mlp":
        H, F = FEED_FORWARD[case["size"]]
        return dict(x=_randn(g, case["tokens"], H), norm_w=(1 + _randn(g, H, scale=0.1)).to(torch.bfloat16),
                    gate=_randn(g, F, H, scale=0.02), up=_randn(g, F, H, scale=0.02), down=_randn(g, H, F, scale=0.02))
    H, F, heads, kv, layers, vocab = MODELS[case["size"]]
    new, _ = _lengths(case)
    sizes = dict(q_proj=(heads * 128, H), k_proj=(kv * 128, H), v_proj=(kv * 128, H), o_proj=(H, heads * 128))
    w = {"model.embed_tokens.weight": _randn(g, vocab, H), "lm_head.weight": _randn(g, vocab, H, scale=0.02),
         "model.norm.weight": (1 + _randn(g, H, scale=0.1)).to(torch.bfloat16)}
    for n in range(layers):
        p = f"model.layers.{n}."
        for name, shape in sizes.items():
            w[f"{p}self_attn.{name}.weight"] = _randn(g, *shape, scale=0.02)
        for name, shape in dict(gate_proj=(F, H), up_proj=(F, H), down_proj=(H, F)).items():
            w[f"{p}mlp.{name}.weight"] = _randn(g, *shape, scale=0.02)
        for name in ("input_layernorm", "post_attention_layernorm"):
            w[f"{p}{name}.weight"] = (1 + _randn(g, H, scale=0.1)).to(torch.bfloat16)
    tokens = torch.randint(0, vocab, (sum(new),), generator=torch.Generator().manual_seed(seed))
    at = _starts(new)
    return dict(new=new, weights=w, prompts=[tokens[a:b].tolist() for a, b in zip(at, at[1:])])


# ----------------------------------------------------------------------------- one pass

def prepare(case, seed):
    s = _inputs(case, seed)
    s["case"] = case
    kind = case["kind"]
    if kind == "attn":
        # split-KV scratch, which a serving process allocates once for its largest decode batch
        from vllm_kunlun_b200.ops.attention_cuda import AttnWorkspace
        s["workspace"] = AttnWorkspace(64, case["heads"], 128, 16, torch.device(DEV, 0))
    elif kind == "mla_prefill":
        s["kv_starts"] = s["qsl"][:-1].contiguous()
    elif kind == "gdn":
        s["cu_host"] = s["cu"].cpu()
    elif kind == "mlp":
        # gate and up rows in the order of the fused projection, laid out once when a model is loaded
        from vllm_kunlun_b200.ops.gemm_cuda import interleave_gate_up
        s["gate_up"] = interleave_gate_up(torch.cat([s.pop("gate"), s.pop("up")]))
    elif kind == "model":
        from vllm_kunlun_b200.config import ModelConfig
        from vllm_kunlun_b200.engine.replay import ScheduleReplay
        H, F, heads, kv, layers, vocab = MODELS[case["size"]]
        cfg = ModelConfig(architecture="LlamaForCausalLM", name="decoder", vocab_size=vocab, hidden_size=H, num_layers=layers,
                          num_heads=heads, num_kv_heads=kv, head_dim=128, intermediate_size=F, rms_norm_eps=1e-5,
                          rope_theta=5e5, max_position=16384)
        tokens = sum(-(-n // BLOCK) * BLOCK for n in s["new"])
        s["replay"] = ScheduleReplay(cfg, "bfloat16", tokens, max_requests=len(s["new"]), block_size=BLOCK, device=DEV)
        with torch.inference_mode():
            s["replay"].engine.runner.model.load_weights(s.pop("weights").items())
    return s


@torch.inference_mode()
def run(s):
    from vllm_kunlun_b200 import ops
    case = s["case"]
    kind = case["kind"]
    if kind == "attn":
        decode = case["new"] == 1
        R = case["requests"]
        return ops.paged_attention(s["q"], s["cache"], s["table"], s["seq_lens"], s["qsl"], s["scale"], max(s["new"]),
                                   max(s["lens"]), case["window"] or None, workspace=s["workspace"],
                                   num_decodes=R if decode else 0, decode_query_len=1, num_decode_tokens=R if decode else 0,
                                   stable_metadata=True)
    if kind == "mla_prefill":
        return ops.mla_prefill_attention(s["q"], s["kv"], s["k_pe"], s["kv_starts"], s["lens"], s["qsl"], True, s["scale"],
                                         max(s["new"]))
    if kind == "mla_decode":
        return ops.mla_attention(s["q"], s["cache"], s["table"], s["seq_lens"], s["qsl"], s["scale"], 512, max(s["new"]),
                                 max(s["lens"]), stable_metadata=True)
    if kind == "gdn":
        Hk, Hv, T, C = case["k_heads"], case["v_heads"], s["T"], s["C"]
        mixed, z = s["qkvz"][:, :C], s["qkvz"][:, C:]
        if max(s["new"]) == 1:
            mixed = ops.causal_conv1d_update(mixed, s["conv_state"], s["conv_w"], None, s["slots"], True, s["init"])
        else:
            mixed = ops.causal_conv1d_fn(mixed, s["conv_w"], None, s["cu"], s["conv_state"], s["slots"], s["init"], True)
        g, beta = ops.fused_gdn_gating(s["A_log"], s["ba"][:, Hv:], s["ba"][:, :Hv], s["dt_bias"])
        kd = Hk * 128
        o = ops.gated_delta_rule(mixed[:, :kd].view(T, Hk, 128), mixed[:, kd:2 * kd].view(T, Hk, 128),
                                 mixed[:, 2 * kd:].view(T, Hv, 128), g, beta, s["states"], s["cu"], s["slots"], s["init"],
                                 128 ** -0.5, True, s["cu_host"])
        o = ops.rms_norm_gated(o.reshape(T * Hv, 128), z.reshape(T * Hv, 128), s["norm_w"], 1e-6, True)
        return o.view(T, Hv * 128), s["states"], s["conv_state"]
    if kind == "moe":
        w, ids = ops.moe_route(s["logits"], s["k"], "softmax", True)
        return ops.fused_moe(s["x"], s["w13"], s["w2"], w, ids, "silu", w13_scale=s["w13_scale"], w2_scale=s["w2_scale"])
    if kind == "mlp":
        x = ops.rmsnorm(s["x"], s["norm_w"], 1e-5)
        return ops.linear(ops.linear_gated_act(x, s["gate_up"], act="silu"), s["down"])
    names = [f"r{i}" for i in range(len(s["prompts"]))]
    return s["replay"].step([dict(id=n, tokens=p, want=[len(p) - 1]) for n, p in zip(names, s["prompts"])], names)


# ----------------------------------------------------------------------------- what a pass cannot do without

def _pairs(case):
    """(query, visible key) pairs of a causal pass, and the cached tokens that it has to read."""
    w = case.get("window", 0)
    pairs = keys = 0
    for n, c in zip(*_lengths(case)):
        seen = [min(p, w) if w else p for p in (c + 1, c + n)]
        if w and c + 1 < w < c + n:
            pairs += (c + 1 + w) * (w - c) // 2 + (c + n - w) * w
        else:
            pairs += (seen[0] + seen[1]) * n // 2
        keys += min(c + n, w + n - 1) if w else c + n
    return pairs, keys


def work(case):
    kind = case["kind"]
    if kind == "attn":
        pairs, keys = _pairs(case)
        T = sum(_lengths(case)[0])
        return dict(flops=4 * 128 * case["heads"] * pairs, bytes=2 * 128 * (2 * T * case["heads"] + 2 * keys * case["kv_heads"]))
    if kind == "mla_prefill":
        pairs, keys = _pairs(case)
        N = case["heads"]
        return dict(flops=2 * (192 + 128) * N * pairs, bytes=2 * keys * (N * (192 + 256 + 128) + 64) + 4 * keys * N)
    if kind == "mla_decode":
        pairs, keys = _pairs(case)
        N = case["heads"]
        return dict(flops=2 * (576 + 512) * N * pairs, bytes=2 * (576 * keys + sum(_lengths(case)[0]) * N * (576 + 512)))
    if kind == "gdn":
        Hv, R, T = case["v_heads"], case["requests"], sum(_lengths(case)[0])
        C = (2 * case["k_heads"] + Hv) * 128
        # per token and head: state times key, rank-one update, state times query; states are read (if carried) and written
        return dict(flops=T * (Hv * 6 * 128 * 128 + 8 * C), bytes=2 * T * (C + 2 * Hv * 128 + 2 * Hv) + 8 * C +
                    (1 + case["carried"]) * R * (4 * Hv * 128 * 128 + 6 * C))
    if kind == "moe":
        H, E, k, I = EXPERTS[case["size"]]
        T = case["tokens"]
        hit = E * (1 - (1 - k / E) ** T)           # experts that T tokens are expected to reach
        return dict(flops=6 * T * k * H * I, bytes=hit * 3 * H * I * (1 if case["fp8"] else 2) + T * (4 * H + 4 * E))
    if kind == "mlp":
        H, F = FEED_FORWARD[case["size"]]
        T = case["tokens"]
        return dict(flops=6 * T * H * F, bytes=2 * (3 * H * F + 2 * T * H))
    H, F, heads, kv, layers, vocab = MODELS[case["size"]]
    T, R = sum(_lengths(case)[0]), case["requests"]
    pairs, _ = _pairs(case)
    layer = H * (2 * heads + 2 * kv) * 128 + 3 * H * F
    return dict(flops=2 * T * layers * layer + 4 * 128 * heads * layers * pairs + 2 * R * H * vocab,
                bytes=2 * (layers * layer + vocab * H + T * H) + 4 * R * vocab)


def tolerance(case):
    """16-bit results of 32-bit sums, rounded again between the steps of a chain."""
    if case["kind"] == "model":
        return {"rel": 3e-2, "max": 0.3}       # four layers of bf16 activations between the sums
    return {"rel": 1e-2, "max": 0.2}


# ----------------------------------------------------------------------------- the same in 64 bits

def _causal(q, k, v, ctx, window, scale):
    """One head: ``q [n, d]``, ``k, v [ctx + n, ...]``, in pieces of queries that fit the memory; also the log-sum-exp."""
    out, lse = [], []
    for a in range(0, q.shape[0], 2048):
        b = min(q.shape[0], a + 2048)
        s = q[a:b] @ k[:ctx + b].T * scale
        pos = torch.arange(ctx + a, ctx + b, device=DEV)[:, None]
        key = torch.arange(ctx + b, device=DEV)[None]
        hide = key > pos
        if window:
            hide |= key <= pos - window
        s.masked_fill_(hide, -math.inf)
        lse.append(torch.logsumexp(s, -1))
        out.append(torch.softmax(s, -1) @ v[:ctx + b])
    return torch.cat(out), torch.cat(lse)


def _delta_rule(i, case):
    """Convolution, gates, recurrence and gated norm of a gated delta net, token by token."""
    Hk, Hv, R, C = case["k_heads"], case["v_heads"], case["requests"], i["C"]
    at, n_max = _starts(i["new"]), max(i["new"])
    slots, carried = i["slots"].long(), i["init"].double()
    x = torch.zeros(R, n_max + 3, C, dtype=torch.float64, device=DEV)
    x[:, :3] = i["conv_state"][slots].double() * carried[:, None, None]
    a_b = torch.zeros(R, n_max, 2 * Hv, dtype=torch.float64, device=DEV)
    for r, n in enumerate(i["new"]):
        x[r, 3:3 + n] = i["qkvz"][at[r]:at[r + 1], :C].double()
        a_b[r, :n] = i["ba"][at[r]:at[r + 1]].double()
    conv_state = i["conv_state"].double()
    for r, n in enumerate(i["new"]):
        conv_state[slots[r]] = x[r, n:n + 3]
    w = i["conv_w"].double()
    y = sum(x[:, j:j + n_max] * w[:, j] for j in range(4))
    y = torch.nn.functional.silu(y)
    kd = Hk * 128
    q, k = (y[..., j * kd:(j + 1) * kd].reshape(R, n_max, Hk, 128) for j in (0, 1))
    v = y[..., 2 * kd:].reshape(R, n_max, Hv, 128)
    q, k = (t * torch.rsqrt((t * t).sum(-1, keepdim=True) + 1e-6) for t in (q, k))
    q, k = (t.repeat_interleave(Hv // Hk, 2) for t in (q * 128 ** -0.5, k))
    beta = torch.sigmoid(a_b[..., :Hv])
    decay = torch.exp(-torch.exp(i["A_log"].double()) * torch.nn.functional.softplus(a_b[..., Hv:] + i["dt_bias"].double()))
    for r, n in enumerate(i["new"]):      # steps behind a request's end leave its state as it is
        beta[r, n:], decay[r, n:] = 0, 1
    S = i["states"].double()[slots] * carried[:, None, None, None]
    o = torch.empty_like(v)
    for t in range(n_max):
        S *= decay[:, t, :, None, None]
        d = beta[:, t, :, None] * (v[:, t] - (S @ k[:, t, :, :, None])[..., 0])
        S += d[..., :, None] * k[:, t, :, None, :]
        o[:, t] = (S @ q[:, t, :, :, None])[..., 0]
    o = torch.cat([o[r, :n] for r, n in enumerate(i["new"])])
    states = i["states"].double()
    states[slots] = S
    z = i["qkvz"][:, C:].double().view(-1, Hv, 128)
    o = o * torch.rsqrt((o * o).mean(-1, keepdim=True) + 1e-6) * i["norm_w"].double() * torch.nn.functional.silu(z)
    return o.reshape(-1, Hv * 128), states, conv_state


def _rms(x, w):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + 1e-5) * w.double()


def _mlp(x, gate, up, down):
    return (torch.nn.functional.silu(x @ gate.double().T) * (x @ up.double().T)) @ down.double().T


def _decoder(i, case):
    H, F, heads, kv, layers, vocab = MODELS[case["size"]]
    w, out = i["weights"], []
    for tokens in i["prompts"]:
        n = len(tokens)
        x = w["model.embed_tokens.weight"][torch.tensor(tokens, device=DEV)].double()
        angle = torch.arange(n, device=DEV).double()[:, None] * 5e5 ** (-torch.arange(64, device=DEV).double() / 64)
        cos, sin = angle.cos()[:, None], angle.sin()[:, None]

        def rotate(t):
            a, b = t[..., :64], t[..., 64:]
            return torch.cat([a * cos - b * sin, b * cos + a * sin], -1)

        for l in range(layers):
            p = f"model.layers.{l}."
            h = _rms(x, w[p + "input_layernorm.weight"])
            q, k, v = (h @ w[f"{p}self_attn.{m}_proj.weight"].double().T for m in "qkv")
            q, k, v = rotate(q.view(n, heads, 128)), rotate(k.view(n, kv, 128)), v.view(n, kv, 128)
            o = torch.stack([_causal(q[:, a], k[:, a * kv // heads], v[:, a * kv // heads], 0, 0, 128 ** -0.5)[0]
                             for a in range(heads)], 1)
            x = x + o.reshape(n, heads * 128) @ w[p + "self_attn.o_proj.weight"].double().T
            h = _rms(x, w[p + "post_attention_layernorm.weight"])
            x = x + _mlp(h, *(w[f"{p}mlp.{m}_proj.weight"] for m in ("gate", "up", "down")))
        out.append(_rms(x[-1:], w["model.norm.weight"]) @ w["lm_head.weight"].double().T)
    return torch.cat(out).cpu()


@torch.inference_mode()
def exact(case, seed):
    i = _inputs(case, seed)
    kind = case["kind"]
    if kind in ("attn", "mla_decode"):
        N, at, out = case["heads"], _starts(i["new"]), []
        for r, (n, total) in enumerate(zip(i["new"], i["lens"])):
            pages = i["cache"][i["table"][r, :-(-total // BLOCK)].long()]
            q = i["q"][at[r]:at[r + 1]].double()
            if kind == "attn":
                kv = pages.transpose(0, 1).transpose(1, 2).reshape(2, case["kv_heads"], -1, 128)[:, :, :total]
                one = lambda h: (kv[0, h * case["kv_heads"] // N].double(), kv[1, h * case["kv_heads"] // N].double())  # noqa: E731
            else:
                rows = pages.reshape(-1, 576)[:total].double()
                one = lambda h: (rows, rows[:, :512])  # noqa: E731
            out.append(torch.stack([_causal(q[:, h], *one(h), total - n, case.get("window", 0), i["scale"])[0] for h in range(N)], 1))
        return torch.cat(out)
    if kind == "mla_prefill":
        N, at, out, lse = case["heads"], _starts(i["new"]), [], []
        for a, b in zip(at, at[1:]):
            kv, pe = i["kv"][a:b].double().view(b - a, N, 256), i["k_pe"][a:b].double()
            got = [_causal(i["q"][a:b, h].double(), torch.cat([kv[:, h, :128], pe], -1), kv[:, h, 128:], 0, 0, i["scale"])
                   for h in range(N)]
            out.append(torch.stack([o for o, _ in got], 1))
            lse.append(torch.stack([m for _, m in got], 1))
        return torch.cat(out), torch.cat(lse)
    if kind == "gdn":
        return _delta_rule(i, case)
    if kind == "moe":
        H, E, k, I = EXPERTS[case["size"]]
        w, ids = torch.softmax(i["logits"].double(), -1).topk(k, -1)
        w = w / w.sum(-1, keepdim=True)
        x, out = i["x"].double(), torch.zeros(case["tokens"], H, dtype=torch.float64, device=DEV)

        def expert(name, e):
            m = i[name][e].double()
            if case["fp8"]:
                m = m * i[name + "_scale"][e].double().repeat_interleave(128, 0).repeat_interleave(128, 1)
            return m

        for e in range(E):
            t, c = (ids == e).nonzero(as_tuple=True)
            if len(t):
                w13 = expert("w13", e)
                out.index_add_(0, t, _mlp(x[t], w13[:I], w13[I:], expert("w2", e)) * w[t, c, None])
        return out
    if kind == "mlp":
        return _mlp(_rms(i["x"].double(), i["norm_w"]), i["gate"], i["up"], i["down"])
    return _decoder(i, case)
