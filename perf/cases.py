"""Performance cases of the quantized decode path: the calls a serving program makes, over the sizes it makes them at.

Three kinds of state. An engine (tenzo_b200.engine.Engine) with its weights and KV cache is what a chat client or a batch
server keeps; the per-kernel calls (tenzo_b200.kernels) are what a program keeps that drives the layers itself, such as the
tensor-parallel decode. Shapes are the repository's own (BitNet-2B and the 8B-shaped model); weights, prompts and caches are
random with the distributions of tenzo_b200.synth.
"""
from __future__ import annotations

import ctypes

import numpy as np
import torch

from tenzo_b200 import abi, kernels, synth
from tenzo_b200.engine import Engine

MODELS = {"2b": synth.BITNET_2B, "8b": synth.SYNTH_8B}
_LIBC = ctypes.CDLL(None)                       # the sampler draws from the process's rand()


def listed():
    return [
        # A chat client's inner loop with the default sampling parameters (temperature, top-k, top-p, repetition penalty
        # over the conversation so far): one token per call, host in and out.
        {"name": "chat_sampled", "kind": "chat", "context": 211, "steps": 8, "sampled": True},
        # Short greedy completion of one sequence with the token fed back on the device (64-token prompt).
        {"name": "chat_greedy", "kind": "chat", "context": 64, "steps": 32, "sampled": False},
        # The same deep into a long conversation.
        {"name": "chat_long", "kind": "chat", "context": 6003, "steps": 4, "sampled": False},
        # Time to the first token: a short question, and a page of text.
        {"name": "prompt_short", "kind": "prompt", "tokens": 64},
        {"name": "prompt_long", "kind": "prompt", "tokens": 1537},
        # A server's decode step: a small group on the block-pool cache; the 8B shape; a full house.
        {"name": "serve_paged_12", "kind": "serve", "model": "2b", "batch": 12, "context": 1500, "steps": 4, "kv_mode": "paged_int8"},
        {"name": "serve_8b_32", "kind": "serve", "model": "8b", "batch": 32, "context": 2048, "steps": 2, "kv_mode": "int8_fused"},
        {"name": "serve_256", "kind": "serve", "model": "2b", "batch": 256, "context": 4096, "steps": 1, "kv_mode": "int8_fused"},
        # One ternary product: the single matrix-vector call, and gate|up with its activation for 256 sequences.
        {"name": "linear_1", "kind": "linear", "rows": 6912, "cols": 2560, "batch": 1, "epilogue": 0, "norm": False},
        {"name": "linear_256", "kind": "linear", "rows": 13824, "cols": 2560, "batch": 256, "epilogue": 2, "norm": True},
        # Attention of one layer for 64 sequences of 8192 keys: in the reference's operation order, and in tolerance mode.
        {"name": "attention_exact", "kind": "attention", "batch": 64, "context": 8192, "ragged": False, "n_q": 20, "n_kv": 5, "mode": 0},
        {"name": "attention_tolerance", "kind": "attention", "batch": 64, "context": 8192, "ragged": False, "n_q": 20, "n_kv": 5, "mode": 1},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    kind = rng.choice(["chat", "prompt", "serve", "serve", "linear", "attention"])
    if kind == "chat":
        context = _log_int(rng, 16, 8000)
        return {"kind": kind, "context": context, "steps": rng.randint(2, 8), "sampled": rng.random() < 0.5}
    if kind == "prompt":
        return {"kind": kind, "tokens": _log_int(rng, 17, 1537)}
    if kind == "serve":
        model = rng.choice(["2b", "2b", "8b"])
        batch = _log_int(rng, 2, 256 if model == "2b" else 64)
        context = _log_int(rng, 100, 4096)
        if model == "8b":                        # a cache of the 8B shape takes 1.7 times the bytes a token
            context = min(context, 131072 // batch)
        kv_mode = rng.choice(["int8_fused", "int8_fused", "paged_int8"])
        if kv_mode == "paged_int8":              # block pools hold fewer sequences, or shorter ones
            context = min(context, 262144 // batch)
        return {"kind": kind, "model": model, "batch": batch, "context": context, "steps": 1 if batch * context > 65536 else 2, "kv_mode": kv_mode}
    if kind == "linear":
        epilogue = rng.randint(0, 2)
        rows = 128 * _log_int(rng, 5, 224)
        cols = 2 * _log_int(rng, 640, 7168)
        if rng.random() < 0.7:                   # model dimensions are mostly multiples of 128
            cols = max(1280, cols // 128 * 128)
        return {"kind": kind, "rows": rows, "cols": cols, "batch": _log_int(rng, 1, 512), "epilogue": epilogue, "norm": rng.random() < 0.7}
    n_q, n_kv = rng.choice([(20, 5), (20, 5), (32, 8), (16, 8), (16, 16)])
    batch = _log_int(rng, 1, 256)
    context = min(_log_int(rng, 64, 16384), 1048576 // batch // (1 if n_kv <= 8 else 2))
    return {"kind": "attention", "batch": batch, "context": context, "ragged": rng.random() < 0.7, "n_q": n_q, "n_kv": n_kv, "mode": rng.randint(0, 1)}


# ---- sizes -------------------------------------------------------------------------------------------------------------
def _lengths(context, batch):
    """Cached tokens of each sequence: spread over (context/2, context], as in a server that admits requests one by one."""
    return [context - (s * 2654435761 >> 7) % max(1, context // 2) for s in range(batch)]


def _round_up(n, m):
    return (n + m - 1) // m * m


def _model_of(case):
    return MODELS[case.get("model", "2b")]


def _weight_bytes(c, logits_steps):
    h, f, kv = c["hidden_size"], c["ffn_dim"], c["num_kv_heads"] * c["head_dim"]
    per_layer = (h * (h + 2 * kv) + h * h + 3 * h * f) // 4 + 4 * (3 * h + f)
    return c["num_layers"] * per_layer + logits_steps * (c["vocab_size"] * (h + 4) + 4 * h)


def _ops_per_token(c):
    h, f, kv = c["hidden_size"], c["ffn_dim"], c["num_kv_heads"] * c["head_dim"]
    return 2 * c["num_layers"] * (h * (h + 2 * kv) + h * h + 3 * h * f)


def _key_bytes(c):
    return c["num_layers"] * c["num_kv_heads"] * (2 * c["head_dim"] + 8)


def _ops_per_key(c):
    return 4 * c["num_layers"] * c["hidden_size"]


# ---- states ------------------------------------------------------------------------------------------------------------
def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _ternary(g, n_bytes):
    """TL1 bytes of independent uniform ternary weights."""
    table = torch.from_numpy(synth._BYTE81).cuda()
    return table[torch.randint(0, 81, (n_bytes,), generator=g, device="cuda", dtype=torch.int32)]


def _host(t):
    out = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    out.copy_(t)
    return out.numpy()


def _engine(case, seed, batch, max_seq, kv_mode="int8_fused"):
    """An engine with random weights, through the public setters."""
    c, g = _model_of(case), _generator(seed)
    e = Engine(batch=batch, **{**c, "max_seq_len": _round_up(max_seq, 16)}, kv_mode=kv_mode.encode())
    h, f = c["hidden_size"], c["ffn_dim"]
    qd, kvd = c["num_q_heads"] * c["head_dim"], c["num_kv_heads"] * c["head_dim"]
    shapes = {"q": (qd, h), "k": (kvd, h), "v": (kvd, h), "out": (h, h), "gate": (f, h), "up": (f, h), "down": (h, f)}
    norms = {"in_norm": h, "attn_sub_norm": h, "post_norm": h, "ffn_sub_norm": f}
    for layer in range(c["num_layers"]):
        w, keep = abi.TenzoLayerWeights(), []
        packed = _host(_ternary(g, sum(n * k // 4 for n, k in shapes.values())))
        weights = _host(1.0 + 0.1 * torch.randn(sum(norms.values()), generator=g, device="cuda"))
        at = 0
        for name, (n, k) in shapes.items():
            keep.append(packed[at: at + n * k // 4])
            setattr(w, name + "_w", keep[-1].ctypes.data_as(abi.c_i8p))
            setattr(w, name + "_scale", 0.016)
            at += n * k // 4
        at = 0
        for name, n in norms.items():
            keep.append(weights[at: at + n])
            setattr(w, name, keep[-1].ctypes.data_as(abi.c_f32p))
            at += n
        assert e.set_layer_weights(layer, w) == abi.SUCCESS
    assert e.set_final_norm(_host(1.0 + 0.1 * torch.randn(h, generator=g, device="cuda"))) == abi.SUCCESS
    table = torch.empty(c["vocab_size"], h, dtype=torch.int8, device="cuda")
    scales = torch.empty(c["vocab_size"], device="cuda")
    for r in range(0, c["vocab_size"], 16384):   # rows of N(0, 0.02^2) values, quantised by their absolute maximum
        rows = 0.02 * torch.randn(min(16384, c["vocab_size"] - r), h, generator=g, device="cuda")
        s = rows.abs().amax(1) / 127
        table[r: r + 16384] = (rows / s[:, None]).round_().to(torch.int8)
        scales[r: r + 16384] = s
    assert e.set_lm_head_i8(_host(table), _host(scales)) == abi.SUCCESS
    return e


def prepare(case, seed):
    return {"chat": _prepare_chat, "prompt": _prepare_prompt, "serve": _prepare_serve, "linear": _prepare_linear,
            "attention": _prepare_attention}[case["kind"]](case, int(seed))


def _prepare_chat(case, seed):
    e = _engine(case, seed, 1, case["context"] + case["steps"] + 1)
    e.kv_fill_random(case["context"], seed=seed)
    past = synth.prompt_tokens(seed, case["context"], 128256)
    params = e.lib.tenzo_default_sampling_params() if case["sampled"] else None
    return {"case": case, "engine": e, "past": past.tolist(), "params": params, "seed": seed}


def _prepare_prompt(case, seed):
    e = _engine(case, seed, 1, case["tokens"] + 8)
    return {"case": case, "engine": e, "prompt": synth.prompt_tokens(seed, case["tokens"], 128256), "params": abi.TenzoSampling(0.0, 0.9, 40, 1.0)}


def _prepare_serve(case, seed):
    e = _engine(case, seed, case["batch"], case["context"] + case["steps"] + 1, case["kv_mode"])
    e.kv_fill_random(case["context"], seed=seed)
    return {"case": case, "engine": e, "lengths": _lengths(case["context"], case["batch"]), "first": synth.prompt_tokens(seed, case["batch"], 128256)}


def _prepare_linear(case, seed):
    g, n, k, b = _generator(seed), case["rows"], case["cols"], case["batch"]
    glu = case["epilogue"] == kernels.EPI_RELU2_GLU
    s = {"case": case, "w": _ternary(g, n * k // 4), "x": torch.randn(b, k, generator=g, device="cuda"), "norm_w": None, "resid": None, "workspace": None}
    if case["norm"]:
        s["norm_w"] = 1.0 + 0.1 * torch.randn(k, generator=g, device="cuda")
    if case["epilogue"] == kernels.EPI_RESIDUAL:
        s["resid"] = torch.randn(b, n, generator=g, device="cuda")
    s["out"] = torch.empty(b, n // 2 if glu else n, device="cuda")
    if b > 1:
        s["workspace"] = torch.empty(kernels.load_library().tenzo_cuda_tl1_gemv_workspace_bytes(b, k), dtype=torch.uint8, device="cuda")
    half = n // 128
    s["scales"], s["seg_ends"] = ([0.016, 0.0161], [half, 2 * half]) if glu else ([0.016], None)
    return s


def _prepare_attention(case, seed):
    g, b, t, nq, nkv = _generator(seed), case["batch"], case["context"], case["n_q"], case["n_kv"]
    rows = _round_up(t, 16)

    def cache():                                 # N(0, 1) rows quantised by their absolute maximum (about 2.7 of 128 values)
        c = torch.empty(b, 1, nkv, rows, 128, dtype=torch.int8, device="cuda")
        for i in range(0, b, 16):
            c[i: i + 16] = (46 * torch.randn(c[i: i + 16].shape, generator=g, device="cuda")).clamp_(-127, 127).round_()
        return c, 0.018 + 0.006 * torch.rand(b, 1, nkv, rows, generator=g, device="cuda")

    s = {"case": case, "rows": rows, "workspace": None}
    s["ck"], s["sk"] = cache()
    s["cv"], s["sv"] = cache()
    for name, heads in (("q", nq), ("k", nkv), ("v", nkv)):
        s[name] = torch.randn(b, heads * 128, generator=g, device="cuda")
    lengths = _lengths(t, b) if case["ragged"] else [t] * b
    s["pos"] = torch.tensor(lengths, dtype=torch.int32, device="cuda") - 1
    cos, sin = np.empty((rows, 64), np.float32), np.empty((rows, 64), np.float32)
    lib = kernels.load_library()
    assert lib.tenzo_ext_rope_tables(rows, 128, 10000.0, cos.ctypes.data_as(abi.c_f32p), sin.ctypes.data_as(abi.c_f32p)) == abi.SUCCESS
    s["cos"], s["sin"] = torch.from_numpy(cos).cuda(), torch.from_numpy(sin).cuda()
    s["out"] = torch.empty(b, nq * 128, device="cuda")
    if case["mode"] == 1:
        s["workspace"] = torch.empty(kernels.attention_workspace_bytes(b, nq, nkv, t), dtype=torch.uint8, device="cuda")
    return s


# ---- one pass ----------------------------------------------------------------------------------------------------------
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "chat":
        e, cur = state["engine"], state["past"][-1]
        e.set_seq_len(0, case["context"])
        if not case["sampled"]:
            return e.decode_greedy([cur], case["steps"])
        _LIBC.srand(state["seed"])
        past = list(state["past"])
        for _ in range(case["steps"]):
            cur = e.generate_step(cur, state["params"], past)
            past.append(cur)
        return np.asarray(past[case["context"]:], np.int32)
    if kind == "prompt":
        e, prompt = state["engine"], state["prompt"]
        e.reset()
        e.prefill_chunk(prompt[:-1])
        token = e.generate_step(int(prompt[-1]), state["params"])
        return {"token": token, "logits": e.read_buffer(15)}
    if kind == "serve":
        e = state["engine"]
        for s, n in enumerate(state["lengths"]):
            e.set_seq_len(s, n)
        return e.decode_greedy(state["first"], case["steps"])
    if kind == "linear":
        return kernels.tl1_gemv(state["x"], state["w"], case["rows"] // 64, case["cols"], state["scales"], state["seg_ends"],
                                epilogue=case["epilogue"], resid=state["resid"], norm_w=state["norm_w"], do_norm=case["norm"],
                                out=state["out"], workspace=state["workspace"])["out"]
    out = kernels.attention_int8(state["q"], state["k"], state["v"], state["ck"], state["cv"], state["sk"], state["sv"], state["pos"], layer=0,
                                 n_q=case["n_q"], n_kv=case["n_kv"], max_seq=state["rows"], rope_cos=state["cos"], rope_sin=state["sin"],
                                 max_len=case["context"], out=state["out"], mode=case["mode"], workspace=state["workspace"])
    return {"out": out, "cache_k": state["ck"], "cache_v": state["cv"], "scale_k": state["sk"], "scale_v": state["sv"]}


def work(case):
    kind = case["kind"]
    if kind == "linear":
        n, k, b = case["rows"], case["cols"], case["batch"]
        n_out = n // 2 if case["epilogue"] == kernels.EPI_RELU2_GLU else n
        vectors = b * (k + n_out * (2 if case["epilogue"] == kernels.EPI_RESIDUAL else 1)) + (k if case["norm"] else 0)
        return {"bytes": n * k // 4 + 4 * vectors, "flops": 2 * n * k * b}
    if kind == "attention":
        b, t = case["batch"], case["context"]
        keys = sum(_lengths(t, b)) if case["ragged"] else b * t
        return {"bytes": keys * case["n_kv"] * 264 + b * 128 * 4 * (2 * case["n_q"] + 2 * case["n_kv"]), "flops": 4 * keys * case["n_q"] * 128}
    c = _model_of(case)
    head = 2 * c["vocab_size"] * c["hidden_size"]
    if kind == "prompt":                         # the layers once over the prompt, the head for its last token
        n = case["tokens"]
        return {"bytes": _weight_bytes(c, 1) + 2 * n * _key_bytes(c) + 4 * c["vocab_size"],
                "flops": n * _ops_per_token(c) + n * (n + 1) // 2 * _ops_per_key(c) + head}
    lengths = [case["context"]] if kind == "chat" else _lengths(case["context"], case["batch"])
    steps, batch = case["steps"], len(lengths)
    keys = sum(n * steps + steps * (steps + 1) // 2 for n in lengths)
    return {"bytes": steps * _weight_bytes(c, 1) + keys * _key_bytes(c), "flops": steps * batch * (_ops_per_token(c) + head) + keys * _ops_per_key(c)}


def tolerance(case):
    # Tolerance-mode attention multiplies in fp16 (weights and queries rounded to 11 bits, fp32 sums). All else reproduces
    # the fp32 operation order of the CPU engine and is the same bit for bit.
    return {"rel": 1e-3} if case["kind"] == "attention" and case["mode"] == 1 else "exact"
