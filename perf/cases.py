"""The workloads whose speed is tracked: what a program that serves GGUF-quantized weights asks of this package.

Every case goes through the package's public entry points: `linear.fused_mul_mat_gguf` (one projection),
`linear.GGUFLinear` (merged projections of one layer), `linear.fused_moe_gguf` (mixture-of-experts feed-forward),
`linear.apply_gguf_embedding` (token embedding) and `sharded.DecoderStack` (a decode step's projections, kept as a CUDA
graph as a serving loop keeps it).  Three things vary: the format mix, the number of tokens and the sizes.

`work` counts wire bytes, activations in and outputs out once each; intermediate activations count as nothing.
"""
import torch

from kaillm_b200 import linear, sharded, synth

DTYPES = {"f32": torch.float32, "f16": torch.float16, "bf16": torch.bfloat16}
CORE = (2, 8, 10, 12, 14, 21)               # Q4_0 Q8_0 Q2_K Q4_K Q6_K IQ3_S: the formats of the benchmark configurations
MORE = (3, 6, 7, 11, 13, 20, 23)            # Q4_1 Q5_0 Q5_1 Q3_K Q5_K IQ4_NL IQ4_XS
I_MATRIX = (20, 21, 23)
LARGEST = 2048 * 5120 * 17408               # token x weight products of the largest listed prefill,
LARGEST_MORE = 333 * 5120 * 6144            # and of the largest one in a format of MORE


def listed():
    return [
        # one projection for one token, called op by op: launches and latency
        {"name": "linear_q4_0_1tok", "kind": "linear", "type": 2, "n": 8192, "k": 2048, "m": 1, "dtype": "f32"},
        # the projections of a decode step, single user and a batch of sixteen: Q8_0 attention, Q4_K gate/up, Q6_K down
        {"name": "stack_1tok", "kind": "stack", "layers": 2, "hidden": 5120, "kv": 1024, "ffn": 17408, "m": 1,
         "t_attn": 8, "t_up": 12, "t_down": 14},
        {"name": "stack_16tok", "kind": "stack", "layers": 2, "hidden": 5120, "kv": 1024, "ffn": 17408, "m": 16,
         "t_attn": 8, "t_up": 12, "t_down": 14},
        # q/k/v of a mixed-type file with a bias, an odd handful of sequences
        {"name": "qkv_mixed_5tok", "kind": "merged", "types": "12,12,14", "rows": "4096,1024,1024", "k": 4096, "m": 5,
         "dtype": "f16"},
        # speculative-decoding verification, 16 sequences x (4 drafted + 1) tokens, on a low-bit file
        {"name": "verify_q2_k_80tok", "kind": "linear", "type": 10, "n": 17408, "k": 5120, "m": 80, "dtype": "bf16"},
        # a decode batch on an i-matrix file: above eight tokens the dispatch reconstructs the weights and multiplies
        {"name": "batch_iq3_s_16tok", "kind": "linear", "type": 21, "n": 17408, "k": 5120, "m": 16, "dtype": "bf16"},
        # a full prefill chunk, and a short prompt of an odd length
        {"name": "prefill_q4_k_2048tok", "kind": "linear", "type": 12, "n": 17408, "k": 5120, "m": 2048, "dtype": "bf16"},
        {"name": "prefill_q5_k_333tok", "kind": "linear", "type": 13, "n": 6144, "k": 5120, "m": 333, "dtype": "f16"},
        # the vocabulary head of a decode batch: one gigabyte of weights for sixteen tokens
        {"name": "lm_head_q6_k_16tok", "kind": "linear", "type": 14, "n": 248320, "k": 5120, "m": 16, "dtype": "bf16"},
        # token embedding of a prefill chunk
        {"name": "embedding_q6_k_2048ids", "kind": "embedding", "type": 14, "n": 248320, "k": 5120, "ids": 2048,
         "dtype": "bf16"},
        # mixture-of-experts feed-forward, 32 experts, top 4: a decode batch and a prefill chunk.  1408 is no multiple of
        # 256, so files of such models hold the down projection in a format of 32-weight blocks
        {"name": "moe_8tok", "kind": "moe", "experts": 32, "top_k": 4, "hidden": 2048, "inter": 1408, "tokens": 8,
         "t_up": 12, "t_down": 8, "dtype": "bf16"},
        {"name": "moe_256tok", "kind": "moe", "experts": 32, "top_k": 4, "hidden": 2048, "inter": 1408, "tokens": 256,
         "t_up": 12, "t_down": 8, "dtype": "bf16"},
    ]


def _log(rng, lo, hi, step=1):
    """A multiple of `step` in [lo, hi], spread over the logarithm."""
    v = lo * (hi / lo) ** rng.random()
    return int(min(hi, max(lo, round(v / step) * step)))


def _k_step(qtype):
    return max(synth.BLOCK[qtype][0], 64)   # 32-weight formats: two blocks, so that rows are not always 256-multiples


def draw(rng):
    kind = rng.choice(("linear", "linear", "prefill", "stack", "stack", "merged", "lm_head", "embedding", "moe", "moe"))
    dtype = rng.choice(("bf16", "bf16", "f16", "f32"))
    if kind in ("linear", "prefill"):
        t = rng.choice(CORE + CORE + MORE)
        k = _log(rng, 1024, 17408, _k_step(t))
        if kind == "linear":
            n = _log(rng, 1024, min(17408, 17408 * 5120 // k))
            return {"kind": "linear", "type": t, "n": n, "k": k, "m": _log(rng, 1, 80), "dtype": dtype}
        m = _log(rng, 81, 2048)
        if t in MORE:
            k = _log(rng, 1024, 5120, _k_step(t))
            m = min(m, LARGEST_MORE // (1024 * k))
        most = LARGEST_MORE if t in MORE else LARGEST
        n = _log(rng, 1024, min(17408, 17408 * 5120 // k, most // (k * m)), 8)
        return {"kind": "linear", "type": t, "n": n, "k": k, "m": m, "dtype": dtype}
    if kind == "stack":
        return {"kind": "stack", "layers": 2, "hidden": _log(rng, 1024, 5120, 256), "kv": rng.choice((256, 512, 1024)),
                "ffn": _log(rng, 2816, 17408, 256), "m": _log(rng, 1, 16), "t_attn": rng.choice((8, 12, 14)),
                "t_up": rng.choice((12, 2, 10)), "t_down": rng.choice((14, 12, 8))}
    if kind == "merged":
        types = rng.choice(("12,12,14", "8,8,8", "13,13,14", "10,10,12", "12,14"))
        rows = [_log(rng, 1024, 8192)] + [_log(rng, 255, 2048)] * (types.count(","))
        return {"kind": "merged", "types": types, "rows": ",".join(map(str, rows)), "k": _log(rng, 1024, 8192, 256),
                "m": _log(rng, 1, 64), "dtype": dtype}
    if kind == "lm_head":
        return {"kind": "linear", "type": rng.choice((14, 8, 12)), "n": _log(rng, 32000, 248320), "k": _log(rng, 1024, 5120, 256),
                "m": _log(rng, 1, 16), "dtype": rng.choice(("bf16", "f16"))}
    if kind == "embedding":
        return {"kind": "embedding", "type": rng.choice((14, 12, 8, 2, 21)), "n": _log(rng, 32000, 248320),
                "k": _log(rng, 1024, 5120, 256), "ids": _log(rng, 1, 2048), "dtype": rng.choice(("bf16", "f16"))}
    t_down = rng.choice((8, 6, 14, 12))
    experts = rng.choice((8, 16, 32, 60, 64))
    return {"kind": "moe", "experts": experts, "top_k": rng.choice((1, 2, 4, 6)), "hidden": _log(rng, 1024, 2048, 256),
            "inter": _log(rng, 512, 1408, 256 if t_down in (12, 14) else 64), "tokens": _log(rng, 1, 160),
            "t_up": rng.choice((12, 8, 10)), "t_down": t_down, "dtype": rng.choice(("bf16", "f16"))}


def _ints(text):
    return [int(v) for v in text.split(",")]


def _scaled(qtype, n, k, seed, dev):
    """Wire rows whose products with unit activations stay near one, as a trained layer's do: every block's fp16 scales
    are brought down (the generator's suit integer tests and would overflow fp16 outputs)."""
    w = synth.wire_torch(qtype, n, k, seed, dev)
    blk, nb = synth.BLOCK[qtype]
    v = w.view(n, k // blk, nb)
    for off in synth.SCALE_FIELDS[qtype]:
        d = v[:, :, off:off + 2].contiguous().view(torch.float16)
        v[:, :, off:off + 2] = (d * (1.0 / 64)).view(torch.uint8)
    return w


def _activations(m, k, dtype, seed, dev):
    g = torch.Generator(device=dev)
    g.manual_seed(seed)
    return torch.randn((m, k), device=dev, generator=g).to(DTYPES[dtype])


def _prepare_stack(case, seed, dev):
    hid, ffn, m = case["hidden"], case["ffn"], case["m"]
    n_qkv = hid + 2 * case["kv"]
    shapes = {"qkv": (case["t_attn"], n_qkv, hid), "o": (case["t_attn"], hid, hid), "gate_up": (case["t_up"], 2 * ffn, hid),
              "down": (case["t_down"], hid, ffn)}
    weights = []
    for layer in range(case["layers"]):
        weights.append({name: (_scaled(t, n, k, seed * 1000 + 10 * layer + i, dev), t, n, k)
                        for i, (name, (t, n, k)) in enumerate(shapes.items())})
    stack = sharded.DecoderStack(weights, m, hid, dev, unsharded=True)
    h = _activations(m, hid, "bf16", seed, dev)
    stream = torch.cuda.Stream(dev)
    stream.wait_stream(torch.cuda.current_stream(dev))
    with torch.cuda.stream(stream):
        stack.forward(h)                     # once outside the capture, as every captured program does
    torch.cuda.current_stream(dev).wait_stream(stream)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = stack.forward(h)
    return {"kind": "stack", "graph": graph, "out": out, "keep": (stack, h)}


def prepare(case, seed):
    dev = torch.device("cuda", torch.cuda.current_device())
    kind = case["kind"]
    if kind == "stack":
        return _prepare_stack(case, seed, dev)
    if kind == "linear":
        return {"kind": kind, "w": _scaled(case["type"], case["n"], case["k"], seed, dev), "type": case["type"],
                "x": _activations(case["m"], case["k"], case["dtype"], seed, dev)}
    if kind == "merged":
        shards = [(_scaled(t, n, case["k"], seed * 10 + i, dev), t)
                  for i, (t, n) in enumerate(zip(_ints(case["types"]), _ints(case["rows"])))]
        layer = linear.GGUFLinear(shards)
        bias = _activations(1, sum(_ints(case["rows"])), case["dtype"], seed + 1, dev).view(-1)
        return {"kind": kind, "layer": layer, "bias": bias, "x": _activations(case["m"], case["k"], case["dtype"], seed, dev)}
    g = torch.Generator(device=dev)
    g.manual_seed(seed)
    if kind == "embedding":
        return {"kind": kind, "w": _scaled(case["type"], case["n"], case["k"], seed, dev), "type": case["type"], "k": case["k"],
                "ids": torch.randint(0, case["n"], (case["ids"],), device=dev, generator=g), "dtype": DTYPES[case["dtype"]]}
    e, hid, inter = case["experts"], case["hidden"], case["inter"]
    w1 = _scaled(case["t_up"], e * 2 * inter, hid, seed * 10, dev).view(e, 2 * inter, -1)
    w2 = _scaled(case["t_down"], e * hid, inter, seed * 10 + 1, dev).view(e, hid, -1)
    router = torch.randn((case["tokens"], e), device=dev, generator=g).softmax(dim=-1)
    weights, ids = router.topk(case["top_k"], dim=-1)
    return {"kind": kind, "w1": w1, "w2": w2, "x": _activations(case["tokens"], hid, case["dtype"], seed, dev),
            "topk_weights": weights / weights.sum(dim=-1, keepdim=True), "topk_ids": ids.to(torch.int32),
            "t_up": case["t_up"], "t_down": case["t_down"]}


def run(state):
    kind = state["kind"]
    if kind == "linear":
        return linear.fused_mul_mat_gguf(state["x"], state["w"], state["type"])
    if kind == "stack":
        state["graph"].replay()
        return state["out"]
    if kind == "merged":
        return state["layer"].apply(state["x"], state["bias"])
    if kind == "embedding":
        return linear.apply_gguf_embedding(state["ids"], state["w"], state["type"], state["k"], state["dtype"])
    return linear.fused_moe_gguf(state["x"], state["w1"], state["w2"], state["topk_weights"], state["topk_ids"],
                                 state["t_up"], state["t_down"])


def _linear_work(qtype, n, k, m, size):
    return synth.weight_bytes(qtype, n, k) + m * (n + k) * size, 2 * m * n * k


def work(case):
    kind = case["kind"]
    size = 4 if case.get("dtype") == "f32" else 2
    if kind == "linear":
        nbytes, flops = _linear_work(case["type"], case["n"], case["k"], case["m"], size)
    elif kind == "merged":
        m, k = case["m"], case["k"]
        parts = list(zip(_ints(case["types"]), _ints(case["rows"])))
        total = sum(n for _, n in parts)
        nbytes = sum(synth.weight_bytes(t, n, k) for t, n in parts) + (m * (k + total) + total) * size
        flops = 2 * m * k * total
    elif kind == "stack":
        hid, ffn, m = case["hidden"], case["ffn"], case["m"]
        n_attn = 2 * hid + 2 * case["kv"]
        per_layer = (synth.weight_bytes(case["t_attn"], n_attn, hid) + synth.weight_bytes(case["t_up"], 2 * ffn, hid) +
                     synth.weight_bytes(case["t_down"], hid, ffn))
        nbytes = case["layers"] * per_layer + 2 * m * hid * size
        flops = case["layers"] * 2 * m * hid * (n_attn + 3 * ffn)
    elif kind == "embedding":
        nbytes = case["ids"] * (synth.row_bytes(case["type"], case["k"]) + case["k"] * size + 8)
        flops = case["ids"] * case["k"]
    else:
        e, k, t = case["experts"], case["top_k"], case["tokens"]
        hid, inter = case["hidden"], case["inter"]
        hit = e * (1 - (1 - k / e) ** t)     # experts that at least one token is routed to
        nbytes = hit * (synth.weight_bytes(case["t_up"], 2 * inter, hid) + synth.weight_bytes(case["t_down"], hid, inter))
        nbytes += 2 * t * hid * size + t * k * 8
        flops = 2 * t * k * 3 * inter * hid
    return {"bytes": nbytes, "flops": flops}


def tolerance(case):
    """Rounding of the output type; where activations pass through q8_1 after a rounding to 16 bits (stack, mixture of
    experts) also the codes that such a rounding tips over.  More than 16 tokens may use fp16 operands."""
    kind = case["kind"]
    if kind == "embedding":
        return "exact"
    if kind in ("stack", "moe"):
        return {"rel": 1e-2, "max": 0.5}
    fine = {"f32": 1e-5, "f16": 1e-3, "bf16": 1e-2}[case["dtype"]]
    fp16_operands = kind == "merged" or case["m"] > 16 or case["type"] in I_MATRIX
    return {"rel": max(fine, 1e-3) if fp16_operands else fine}
