"""What the speed of this framework is measured on: the layers and blocks that its decoders run, each through the entry point that a
program calls, over the sizes at which it is called.

The int4 decoder: its linear layer in the draft mode (W4A4, packed int4 activations or one int4 value per byte) and in the verify mode
(W4A16), from single tokens to prompt portions, on the shapes of Llama-3-8B / 70B and Qwen2.5-14B; the rotation in front of down_proj
with SiLU and the quantiser; its attention over the KV cache for decoding, speculative verification and prompt portions; a whole
verify-mode pass of a model. The sequence-mixer library: the window attention, the routed experts and the gated recurrence of its models.

A case is a dict of plain values; `kind` says which of the blocks below it is.
"""
import math

import torch

LINEAR_SHAPES = [  # (N, K) of qkv, o, gate_up and down of Llama-3-8B, Qwen2.5-14B and Llama-3-70B; o of 8B is also its q_proj
    (6144, 4096), (4096, 4096), (28672, 4096), (4096, 14336), (7168, 5120), (27648, 5120), (10240, 8192), (8192, 8192)]
F64 = torch.float64


def listed():
    return [
        # q_proj of Llama-3-8B for the four sequences of an interactive server: one draft token each. The smallest call.
        {"name": "draft_linear_4", "kind": "linear", "mode": "w4a4", "m": 4, "n": 4096, "k": 4096, "bias": False},
        # gate_up for 64 concurrent sequences in a draft pass, activations one int4 value per byte as the decoder passes them there
        {"name": "draft_linear_64", "kind": "linear", "mode": "w4a4_bytes", "m": 64, "n": 28672, "k": 4096, "bias": False},
        # down_proj when four sequences verify three draft tokens each
        {"name": "verify_linear_16", "kind": "linear", "mode": "w4a16", "m": 16, "n": 4096, "k": 14336, "bias": False},
        # gate_up when 64 sequences verify three draft tokens each
        {"name": "verify_linear_256", "kind": "linear", "mode": "w4a16", "m": 256, "n": 28672, "k": 4096, "bias": False},
        # qkv_proj of Llama-3-70B for a long prompt portion of ragged length
        {"name": "prompt_linear_1999", "kind": "linear", "mode": "w4a16", "m": 1999, "n": 10240, "k": 8192, "bias": False},
        # between gate_up and down_proj of a draft pass for 64 sequences: SiLU, rotation, int4 values and scales
        {"name": "rotate_quant_64", "kind": "rotate", "rows": 64, "n": 512, "quant": True},
        # the verify pass of 64 sequences x 4 tokens over unequal contexts
        {"name": "attention_verify_256", "kind": "attention", "seqs": 64, "per": 4, "context": 900, "cache": 1024, "heads": 32, "kv": 8},
        # a prompt portion in the middle of a prompt, one sequence
        {"name": "attention_prompt_1000", "kind": "attention", "seqs": 1, "per": 1000, "context": 1000, "cache": 2048, "heads": 32, "kv": 8},
        # a whole verify-mode pass: a prompt of 509 tokens through two layers of Llama-3-8B's sizes, and the last token's logits
        {"name": "pass_prompt_509", "kind": "pass", "seqs": 1, "per": 509, "context": 0, "layers": 2, "cache": 1024},
        # window attention with sinks and an output gate, a prompt portion of 2000 tokens of one sequence
        {"name": "window_prompt_2000", "kind": "window", "seqs": 1, "per": 2000, "context": 1100, "window": 1024, "heads": 16, "kv": 4},
        # routed experts of a prompt portion
        {"name": "experts_2048", "kind": "experts", "tokens": 2048, "width": 2048, "ff": 1024, "experts": 16, "top": 4},
        # the gated recurrence of a prompt portion
        {"name": "scan_prompt_1500", "kind": "scan", "seqs": 1, "per": 1500, "heads": 16, "dim": 128},
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["linear", "linear", "linear", "linear", "rotate", "attention", "attention", "pass", "window", "experts", "scan"])
    if kind == "linear":
        mode = rng.choice(["w4a4", "w4a4_bytes", "w4a16", "w4a16"])
        n, k = rng.choice(LINEAR_SHAPES)
        most = {"w4a4": 256, "w4a4_bytes": 256, "w4a16": 2000}[mode]
        m = log(48 if mode == "w4a4_bytes" else 1, min(most, 1999 * 10240 * 8192 // (n * k)))
        return {"kind": kind, "mode": mode, "m": m, "n": n, "k": k, "bias": rng.random() < 0.25}
    if kind == "rotate":
        return {"kind": kind, "rows": log(1, 512), "n": rng.choice([128, 256, 512, 1024]), "quant": rng.random() < 0.5}
    if kind == "attention":
        heads, kv = rng.choice([(32, 8), (32, 8), (16, 4), (64, 8), (40, 8)])
        if rng.random() < 0.5:  # one token, or a draft's tokens, of many sequences
            seqs, per = log(1, 64), rng.choice([1, 2, 4, 5])
            cache = rng.choice([512, 1024, 2048])
            return {"kind": kind, "seqs": seqs, "per": per, "context": rng.randint(40, cache - 8), "cache": cache, "heads": heads, "kv": kv}
        seqs, per = rng.choice([1, 1, 2, 3]), log(40, 1000 * 32 // heads // 2)
        cache = rng.choice([1024, 2048, 4096])
        context = rng.randint(0, min(cache - per, 1000))
        return {"kind": kind, "seqs": seqs, "per": per, "context": context, "cache": cache, "heads": heads, "kv": kv}
    if kind == "pass":
        per = log(1, 500)
        return {"kind": kind, "seqs": 1 if per > 64 else rng.randint(1, max(1, 64 // per)), "per": per, "context": rng.randint(0, 400), "layers": rng.choice([1, 2]),
                "cache": 1024}
    if kind == "window":
        heads, kv = rng.choice([(16, 4), (32, 8), (16, 2)])
        if rng.random() < 0.4:
            return {"kind": kind, "seqs": log(1, 64), "per": 1, "context": rng.randint(1, 1500), "window": rng.choice([128, 512, 1024]), "heads": heads, "kv": kv}
        return {"kind": kind, "seqs": rng.choice([1, 1, 2, 4]), "per": log(64, 480 * 16 // heads), "context": rng.randint(0, 1500),
                "window": rng.choice([100, 512, 1024, 2048]), "heads": heads, "kv": kv}
    if kind == "experts":
        width, ff, experts, top = rng.choice([(2048, 1024, 16, 4), (4096, 2048, 8, 2), (1024, 512, 32, 6)])
        return {"kind": kind, "tokens": log(32, 2048 if width == 2048 else 1024), "width": width, "ff": ff, "experts": experts, "top": top}
    heads, dim = rng.choice([(16, 128), (32, 128), (8, 64), (16, 64)])
    return {"kind": kind, "seqs": rng.choice([1, 1, 2, 5]), "per": log(20, 1500 * 16 // heads // 5), "heads": heads, "dim": dim}


# ---- inputs -------------------------------------------------------------------------------------------------------------------------
def _gen(seed, part):
    return torch.Generator(device="cuda").manual_seed(seed * 1009 + part)


def _normal(g, *shape, dtype=torch.float16, scale=1.0):
    return (torch.randn(*shape, generator=g, device="cuda") * scale).to(dtype)


def _contexts(case, seed):
    """How many tokens each sequence holds before the pass: unequal where there are several."""
    most = case["context"]
    if case["seqs"] == 1:
        return [most]
    g = torch.Generator().manual_seed(seed * 31 + 5)
    return torch.randint(most // 2, most + 1, (case["seqs"],), generator=g).tolist()


def _positions(case, seed):
    first = _contexts(case, seed)
    pos = torch.cat([torch.arange(f, f + case["per"]) for f in first]).to(torch.int32)
    seq = torch.arange(case["seqs"]).repeat_interleave(case["per"]).to(torch.int32)
    return first, pos, seq


def _weight(seed, n, k):
    """Packed int4 weights [n, k / 2] (two signed values per byte, the even one in the low half) and scales [n]."""
    g = _gen(seed, 1)
    w = torch.randint(0, 256, (n, k // 2), generator=g, dtype=torch.uint8, device="cuda").view(torch.int8)
    scales = ((0.5 + torch.rand(n, generator=g, device="cuda")) * 2.0 ** -7).to(torch.float16)
    return w, scales


def _linear_inputs(case, seed):
    m, n, k = case["m"], case["n"], case["k"]
    w, scales = _weight(seed, n, k)
    g = _gen(seed, 2)
    bias = _normal(g, n, scale=0.1) if case["bias"] else None
    x = _normal(g, m, k)  # a normed row
    if case["mode"] == "w4a16":
        return w, scales, bias, x, None, None
    amax = x.float().abs().amax(1, keepdim=True)
    q = (x.float() * (7.0 / amax)).round().clamp(-8, 7).to(torch.int8)
    return w, scales, bias, x, q, (amax[:, 0] / 7.0).to(torch.float16)


def _rotate_inputs(case, seed):
    gate_up = _normal(_gen(seed, 1), case["rows"], 2 * 28 * case["n"])
    return gate_up, 1.0 / math.sqrt(28 * case["n"])


def _attention_inputs(case, seed):
    first, pos, seq = _positions(case, seed)
    g = _gen(seed, 1)
    heads, kv, t = case["heads"], case["kv"], case["seqs"] * case["per"]
    qkv = _normal(g, t, (heads + 2 * kv) * 128)  # queries after the rotary embedding
    keys = _normal(g, case["seqs"], case["cache"], kv, 128)
    values = _normal(g, case["seqs"], case["cache"], kv, 128)
    return first, pos, seq, qkv, keys, values


def _window_inputs(case, seed):
    first, pos, seq = _positions(case, seed)
    g = _gen(seed, 1)
    heads, kv, t = case["heads"], case["kv"], case["seqs"] * case["per"]
    cap = case["window"] - 1 + t
    q = _normal(g, t, heads, 128, dtype=torch.float32)
    keys = _normal(g, case["seqs"], cap, kv, 128, dtype=torch.bfloat16)
    values = _normal(g, case["seqs"], cap, kv, 128, dtype=torch.bfloat16)
    sink = _normal(g, heads, dtype=torch.float32)
    gate = _normal(g, t, heads * 128, dtype=torch.bfloat16)
    return first, pos, seq, q, keys, values, sink, gate


def _experts_inputs(case, seed):
    t, w, f, e = case["tokens"], case["width"], case["ff"], case["experts"]
    g = _gen(seed, 1)
    h = _normal(g, t, w, dtype=torch.bfloat16)
    gate_up = _normal(g, e, 2 * f, w, dtype=torch.bfloat16, scale=w ** -0.5)
    down = _normal(g, e, w, f, dtype=torch.bfloat16, scale=f ** -0.5)
    # a router's choices: some experts are asked for more often than others
    score = torch.randn(t, e, generator=g, device="cuda") + 0.7 * torch.randn(e, generator=g, device="cuda")
    return h, gate_up, down, score.topk(case["top"], 1).indices.to(torch.int32).contiguous()


def _scan_inputs(case, seed):
    heads, dim, t = case["heads"], case["dim"], case["seqs"] * case["per"]
    g = _gen(seed, 1)
    p = _normal(g, t, 3 * heads * dim, dtype=torch.bfloat16)  # [q | f | v] as projected
    bias = _normal(g, heads * dim, dtype=torch.float32) + 2.0
    lower = torch.rand(heads * dim, generator=g, device="cuda") * 0.5
    norm = 1.0 + _normal(g, dim, dtype=torch.float32, scale=0.1)
    return p, bias, lower, norm


def _table(case, seed):
    """The step table that the scheduler hands to the sequence-mixer models: slot, position, segment begin and end, tail phase."""
    first, pos, seq = _positions(case, seed)
    per = case["per"]
    begin = seq * per
    return torch.stack([seq, pos, begin, begin + per, torch.zeros_like(seq)]).to(torch.int32).cuda()


def _config(case):
    from qspec_b200.model import QSpecLlamaConfig
    return QSpecLlamaConfig.llama3_8b(num_hidden_layers=case["layers"], vocab_size=32000, max_seq_len=case["cache"])


def prepare(case, seed):
    kind = case["kind"]
    if kind == "linear":
        from qspec_b200.nn import Linear4bit, PackedQuantizedTensor
        w, scales, bias, x, q, s = _linear_inputs(case, seed)
        layer = Linear4bit(case["k"], case["n"], device="cuda", empty_init=True)
        layer.weight, layer.weight_scales, layer.bias = w, scales, bias
        if case["mode"] == "w4a4":
            x = PackedQuantizedTensor(((q[:, 0::2] & 15) | (q[:, 1::2] << 4)).contiguous(), s)
        elif case["mode"] == "w4a4_bytes":
            x = PackedQuantizedTensor(q, s)
        how = {"w4a4": {"w4a4": True}, "w4a4_bytes": {"w4a8": True}, "w4a16": {}}[case["mode"]]
        return {"kind": kind, "layer": layer, "x": x, "how": how, "out": torch.empty(case["m"], case["n"], dtype=torch.float16, device="cuda")}
    if kind == "rotate":
        gate_up, scale = _rotate_inputs(case, seed)
        rows, width = case["rows"], 28 * case["n"]
        state = {"kind": kind, "gate_up": gate_up, "n": case["n"], "scale": scale, "out": None, "out_q": None, "scales": None}
        if case["quant"]:
            state["out_q"] = torch.empty(rows, width // 2, dtype=torch.int8, device="cuda")
            state["scales"] = torch.empty(rows, dtype=torch.float16, device="cuda")
        else:
            state["out"] = torch.empty(rows, width, dtype=torch.float16, device="cuda")
        return state
    if kind == "attention":
        _, pos, seq, qkv, keys, values = _attention_inputs(case, seed)
        out = torch.empty(qkv.shape[0], case["heads"] * 128, dtype=torch.float16, device="cuda")
        return {"kind": kind, "qkv": qkv, "keys": keys, "values": values, "pos": pos.cuda(), "seq": seq.cuda(), "out": out, "heads": case["heads"], "kv": case["kv"]}
    if kind == "pass":
        from qspec_b200.model import QSpecLlamaModel
        _, pos, seq = _positions(case, seed)
        t = pos.numel()
        g = _gen(seed, 1)
        ids = torch.randint(0, 32000, (t,), generator=g, device="cuda")
        model = QSpecLlamaModel(_config(case), max_batch=case["seqs"], max_tokens=max(t, 16), seed=seed)
        for cache in (model.cache_k, model.cache_v):
            cache.copy_(_normal(g, *cache.shape))
        last = (torch.arange(1, case["seqs"] + 1) * case["per"] - 1).cuda()
        return {"kind": kind, "model": model, "ids": ids, "pos": pos.cuda(), "seq": seq.cuda(), "last": last}
    if kind == "window":
        _, _, _, q, keys, values, sink, gate = _window_inputs(case, seed)
        out = torch.empty(q.shape[0], case["heads"], 128, dtype=torch.bfloat16, device="cuda")
        return {"kind": kind, "q": q, "keys": keys, "values": values, "sink": sink, "gate": gate, "out": out, "table": _table(case, seed), "window": case["window"],
                "rows": case["per"] >= 16}
    if kind == "experts":
        h, gate_up, down, chosen = _experts_inputs(case, seed)
        out = torch.empty(case["tokens"], case["top"], case["width"], dtype=torch.bfloat16, device="cuda")
        return {"kind": kind, "h": h, "gate_up": gate_up, "down": down, "chosen": chosen, "out": out, "experts": case["experts"], "ff": case["ff"]}
    p, bias, lower, norm = _scan_inputs(case, seed)
    heads, dim, t = case["heads"], case["dim"], p.shape[0]
    table = _table(dict(case, context=0), seed)
    return {"kind": kind, "p": p, "bias": bias, "lower": lower, "norm": norm, "heads": heads, "dim": dim, "table": table,
            "starts": (torch.arange(case["seqs"]) * case["per"]).to(torch.int32).cuda(),
            "state": torch.zeros(case["seqs"], heads, dim, dim, device="cuda"), "scratch": torch.empty(t * heads * 4 * dim, device="cuda"),
            "out": torch.empty(t, heads * dim, dtype=torch.bfloat16, device="cuda")}


def run(state):
    from qspec_b200 import ops
    s, kind = state, state["kind"]
    if kind == "linear":
        return s["layer"](s["x"], s["out"], **s["how"])
    if kind == "rotate":
        ops.hadamard_k28(None, s["n"], s["scale"], gate_up=s["gate_up"], out=s["out"], out_q=s["out_q"], scale_out=s["scales"])
        return s["out"] if s["out"] is not None else (s["out_q"], s["scales"])
    if kind == "attention":
        heads, kv = s["heads"], s["kv"]
        t = s["pos"].numel()
        # the decoder's own choice between its two forms
        call = ops.seq_attention if t >= 32 and ops.seq_attention_supported(t, heads, kv, 128, s["keys"].shape[1]) else ops.decode_attention
        return call(s["qkv"], s["keys"], s["values"], s["pos"], s["seq"], s["out"], heads, kv, 128, 128 ** -0.5)
    if kind == "pass":
        m = s["model"]
        hidden = m.forward(s["ids"], s["pos"], s["seq"], w4a4=False)
        return hidden, m.logits(hidden.index_select(0, s["last"])), m.cache_k, m.cache_v
    if kind == "window":
        ops.seq_window_attention_mma(s["q"], s["keys"], None, s["values"], s["out"], s["table"], s["window"], 128 ** -0.5, s["rows"], sink=s["sink"], gate=s["gate"])
        return s["out"]
    if kind == "experts":
        ops.moe_expert_grouped(s["h"], s["gate_up"], s["down"], s["chosen"], s["out"], s["experts"], s["ff"], 0.0, act="silu")
        return s["out"]
    ops.seq_hgrn2(s["p"], s["bias"], s["lower"], s["norm"], s["state"], s["scratch"], s["out"], s["table"], s["heads"], s["dim"], s["dim"], 1e-5, seg_starts=s["starts"])
    return s["out"], s["state"]


# ---- what a pass cannot do without ------------------------------------------------------------------------------------------------
def _pairs(case, window=1 << 30):
    """Visible (query, key) pairs, and the keys that a pass reads, with every sequence at the middle of its contexts."""
    n, first = case["seqs"], case["context"] if case["seqs"] == 1 else case["context"] * 3 // 4
    pairs = sum(min(first + i + 1, window) for i in range(case["per"]))
    return n * pairs, n * min(first + case["per"], window - 1 + case["per"])


def work(case):
    kind = case["kind"]
    if kind == "linear":
        m, n, k = case["m"], case["n"], case["k"]
        act = {"w4a4": k // 2 + 2, "w4a4_bytes": k + 2, "w4a16": 2 * k}[case["mode"]]
        return {"bytes": n * k // 2 + 2 * n * (2 if case["bias"] else 1) + m * act + 2 * m * n, "flops": 2 * m * n * k}
    if kind == "rotate":
        rows, k = case["rows"], 28 * case["n"]
        return {"bytes": rows * (4 * k + (k // 2 + 2 if case["quant"] else 2 * k)), "flops": rows * k * (28 + int(math.log2(case["n"])) + 6)}
    if kind in ("attention", "window"):
        pairs, keys = _pairs(case, case.get("window", 1 << 30))
        t, heads, kv = case["seqs"] * case["per"], case["heads"], case["kv"]
        rows = t * heads * 128 * ((2 + 2) if kind == "attention" else (4 + 2 + 2))
        return {"bytes": keys * kv * 128 * 4 + rows, "flops": 4 * pairs * heads * 128}
    if kind == "pass":
        t, layers = case["seqs"] * case["per"], case["layers"]
        pairs, keys = _pairs(case)
        weights = 6144 * 4096 + 4096 * 4096 + 28672 * 4096 + 4096 * 14336
        head = 32000 * 4096
        return {"bytes": layers * (weights // 2 + keys * 8 * 128 * 4) + 2 * head + t * 4096 * 4 + case["seqs"] * 64000,
                "flops": layers * (2 * t * weights + 4 * pairs * 32 * 128) + 2 * case["seqs"] * head}
    if kind == "experts":
        t, w, f, e, top = (case[i] for i in ("tokens", "width", "ff", "experts", "top"))
        return {"bytes": min(e, t * top) * 3 * w * f * 2 + t * (w * 2 + top * (w * 2 + 4)), "flops": 6 * t * top * w * f}
    t, heads, dim = case["seqs"] * case["per"], case["heads"], case["dim"]
    return {"bytes": t * heads * dim * 8 + case["seqs"] * heads * dim * dim * 4, "flops": t * heads * dim * dim * 5}


def tolerance(case):
    """About four times what one pass differs by from the same in 64 bits, which is mostly the rounding of the outputs."""
    kind = case["kind"]
    if kind == "linear":
        # whole-number sums and one order of the scale factors: every correct implementation gives the same float16 values
        return {"rel": 8e-4} if case["mode"] == "w4a16" else "exact"
    if kind == "rotate":
        # float16 roundings after SiLU and after the first rotation; a value on the edge between two steps of the quantiser may fall either way
        return {"rel": 1.3e-3, "differ": 0.005}
    if kind == "attention":
        return {"rel": 8e-4}
    if kind == "pass":  # float16 roundings of every layer travel through those that follow
        return {"rel": 1.2e-2}
    if kind == "window":  # bfloat16 outputs, queries rounded to bfloat16 for the product
        return {"rel": 1e-2}
    if kind == "experts":  # bfloat16 activations between the two products
        return {"rel": 1.4e-2}
    return {"rel": 7e-3}


# ---- the same in 64 bits ----------------------------------------------------------------------------------------------------------
def _int4(w, dtype=F64):
    """Signed int4 values [n, k] of packed bytes [n, k / 2]."""
    low = (w << 4) >> 4
    return torch.stack((low, w >> 4), -1).reshape(w.shape[0], -1).to(dtype)


def _had28():
    """The 28 x 28 Hadamard matrix of Paley's second construction over the field of 13 elements."""
    squares = {i * i % 13 for i in range(1, 13)}
    c = torch.ones(14, 14, dtype=F64)
    c[0, 0] = 0
    for i in range(13):
        for j in range(13):
            c[i + 1, j + 1] = 0 if i == j else 1 if (j - i) % 13 in squares else -1
    one = torch.eye(14, dtype=F64)
    return torch.cat((torch.cat((c + one, c - one), 1), torch.cat((c - one, -c - one), 1)), 0).cuda()


def _hadamard(n):
    h = torch.ones(1, 1, dtype=F64)
    while h.shape[0] < n:
        h = torch.cat((torch.cat((h, h), 1), torch.cat((h, -h), 1)), 0)
    return h.cuda()


def _rotated(gate_up, n):
    k = 28 * n
    up, gate = gate_up[:, :k].to(F64), gate_up[:, k:].to(F64)
    a = gate * torch.sigmoid(gate) * up
    return (_had28() @ (a.view(-1, 28, n) @ _hadamard(n))).reshape(-1, k)


def _softmax_rows(q, keys, values, first, rows, begin, scale, window, sink):
    """One sequence: q [t, heads, d] at positions first .., keys / values [positions from `begin`, kv, d]."""
    t, heads = q.shape[:2]
    rep = heads // keys.shape[1]
    out = []
    i = torch.arange(first, first + t, device="cuda")[:, None]
    j = torch.arange(begin, begin + rows, device="cuda")[None, :]
    hidden = (j > i) | (i - j >= window)
    for h in range(heads):
        s = (q[:, h].to(F64) @ keys[:, h // rep].to(F64).T) * scale
        s = s.masked_fill(hidden, -math.inf)
        if sink is not None:
            s = torch.cat((s, sink[h].to(F64).expand(t, 1)), 1)
        p = torch.softmax(s, 1)[:, :rows]
        out.append(p @ values[:, h // rep].to(F64))
    return torch.stack(out, 1)


def _exact_pass(case, seed):
    state = prepare(case, seed)
    m, cfg = state["model"], _config(case)
    first, pos, seq = _positions(case, seed)
    t, eps = pos.numel(), cfg.rms_norm_eps
    inv = cfg.rope_theta ** (-torch.arange(0, 128, 2, dtype=torch.float32) / 128)
    angle = torch.outer(torch.arange(case["cache"], dtype=torch.float32), inv).cuda()
    cos, sin = angle.cos().half().to(F64)[pos.long().cuda()][:, None], angle.sin().half().to(F64)[pos.long().cuda()][:, None]
    ck, cv = m.cache_k.to(F64), m.cache_v.to(F64)

    def norm(x):
        y = x - x.mean(1, keepdim=True)
        return y / torch.sqrt((y * y).mean(1, keepdim=True) + eps)

    def linear(x, layer):
        return x @ _int4(layer.weight.view(torch.int8)).T * layer.weight_scales.view(-1).to(F64)

    def turn(x):
        a, b = x[..., :64], x[..., 64:]
        return torch.cat((a * cos - b * sin, b * cos + a * sin), -1)

    x = m.embed[state["ids"]].to(F64)
    for i, layer in enumerate(m.layers):
        qkv = linear(norm(x), layer.qkv_proj).view(t, 48, 128)
        q, k, v = turn(qkv[:, :32]), turn(qkv[:, 32:40]), qkv[:, 40:]
        ck[i, state["seq"].long(), state["pos"].long()] = k
        cv[i, state["seq"].long(), state["pos"].long()] = v
        per = case["per"]
        a = torch.cat([_softmax_rows(q[b * per:(b + 1) * per], ck[i, b, :f + per], cv[i, b, :f + per], f, f + per, 0, 128 ** -0.5, 1 << 30, None) for b, f in enumerate(first)])
        x = x + linear((_hadamard(32) @ a).reshape(t, 4096) * m.scale_heads, layer.o_proj)
        x = x + linear(_rotated(linear(norm(x), layer.gate_up), 512) * m.scale_mlp, layer.down_proj)
    hidden = norm(x)
    return hidden, hidden[state["last"]] @ m.lm_head.to(F64).T, ck, cv


def exact(case, seed):
    kind = case["kind"]
    if kind == "linear":
        w, scales, bias, x, q, s = _linear_inputs(case, seed)
        y = (x if q is None else q).to(F64) @ _int4(w).T
        if s is not None:
            y = y * s.to(F64)[:, None]
        y = y * scales.to(F64)
        return y if bias is None else y + bias.to(F64)
    if kind == "rotate":
        gate_up, scale = _rotate_inputs(case, seed)
        y = _rotated(gate_up, case["n"]) * scale
        if not case["quant"]:
            return y
        return None, y.abs().amax(1) / 7.0
    if kind == "attention":
        first, pos, seq, qkv, keys, values = _attention_inputs(case, seed)
        per, heads = case["per"], case["heads"]
        q = qkv[:, :heads * 128].view(-1, heads, 128)
        out = [_softmax_rows(q[b * per:(b + 1) * per], keys[b, :f + per], values[b, :f + per], f, f + per, 0, 128 ** -0.5, 1 << 30, None) for b, f in enumerate(first)]
        return torch.cat(out).reshape(-1, heads * 128)
    if kind == "pass":
        return _exact_pass(case, seed)
    if kind == "window":
        first, pos, seq, q, keys, values, sink, gate = _window_inputs(case, seed)
        per, cap, out = case["per"], keys.shape[1], []
        for b, f in enumerate(first):
            begin = max(0, f + 1 - case["window"])
            ring = torch.arange(begin, f + per, device="cuda") % cap
            out.append(_softmax_rows(q[b * per:(b + 1) * per], keys[b, ring], values[b, ring], f, f + per - begin, begin, 128 ** -0.5, case["window"], sink))
        return torch.cat(out) * torch.sigmoid(gate.to(F64)).view(-1, case["heads"], 128)
    if kind == "experts":
        h, gate_up, down, chosen = _experts_inputs(case, seed)
        f = case["ff"]
        out = torch.empty(case["tokens"], case["top"], case["width"], dtype=F64, device="cuda")
        for e in range(case["experts"]):
            t, c = (chosen == e).nonzero(as_tuple=True)
            z = h[t].to(F64) @ gate_up[e].to(F64).T
            g = z[:, :f]
            out[t, c] = (g * torch.sigmoid(g) * z[:, f:]) @ down[e].to(F64).T
        return out
    p, bias, lower, norm = _scan_inputs(case, seed)
    heads, dim, per = case["heads"], case["dim"], case["per"]
    z = p.to(F64).view(case["seqs"], per, 3, heads, dim)
    q = z[:, :, 0] * torch.sigmoid(z[:, :, 0])
    low = lower.to(F64).view(heads, dim)
    f = low + (1.0 - low) * torch.sigmoid(z[:, :, 1] + bias.to(F64).view(heads, dim))
    state = torch.zeros(case["seqs"], heads, dim, dim, dtype=F64, device="cuda")
    out = []
    for t in range(per):
        state = f[:, t, :, :, None] * state + (1.0 - f[:, t])[..., None] * z[:, t, 2][:, :, None, :]
        out.append((q[:, t, :, None] @ state)[:, :, 0])
    o = torch.stack(out, 1)
    o = o / torch.sqrt((o * o).mean(-1, keepdim=True) + 1e-5) * norm.to(F64)
    return o.reshape(-1, heads * dim), state
