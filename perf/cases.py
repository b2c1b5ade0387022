"""The work whose speed counts: what users of this framework have it do, through its public entry points, over the sizes they use.

    listed()            the cases with names                 draw(rng)            one more case of the same ranges
    prepare(case, seed) what a program has before the call   run(state)           one pass, its outputs
    work(case)          bytes and operations of one pass     tolerance(case)      what two correct implementations may differ by
    exact(case, seed)   the outputs in 64 bits, from plain torch

A case is a dict of plain values; ``kind`` says which of five uses it stands for:

    operator   one DequantMatMul: the fused operator of the engine's own graphs
    w8a8       DynamicQuantizeLinear and QuantizedMatMul, the engine's W8A8 pair, over a prompt's activations
    step       one decode step of a batch of sequences that have a long context (a server's inner loop); on the device or, ``host``,
               with token ids and logits in host memory (the engine's own session)
    stream     one step of an endless conversation in the streaming (sink + ring) cache, long after the ring has wrapped
    request    prompts in prefill chunks and a few decode steps behind them, of any model family (``family``)
"""
from __future__ import annotations

import math

import numpy as np
import torch

from my_nn_engine_b200 import fimadra, ops, vebisun
from my_nn_engine_b200.decoder import DecoderModel

DTYPES = {"bf16": torch.bfloat16, "f16": torch.float16, "f32": torch.float32}

# Architectures of this repository's benchmark (random weights; there are no checkpoints here).
LLAMA = {
    "llama3-8b": dict(hidden_size=4096, num_hidden_layers=32, num_attention_heads=32, num_key_value_heads=8, head_dim=128,
                      intermediate_size=14336, vocab_size=128256, rms_norm_eps=1e-5, rope_theta=500000.0),
    "tinyllama": dict(hidden_size=2048, num_hidden_layers=22, num_attention_heads=32, num_key_value_heads=4, head_dim=64,
                      intermediate_size=5632, vocab_size=32000, rms_norm_eps=1e-5, rope_theta=10000.0),
}
VEBISUN = {
    "small-experts": dict(width=2048, heads=32, kv=8, dim=128, window=1024, experts=64, top=8, ff=1024, groups=8, keep=4, layers=8, vocab=32000),
    "large-experts": dict(width=4096, heads=32, kv=8, dim=128, window=4096, experts=8, top=2, ff=7168, groups=4, keep=2, layers=4, vocab=32000),
}
FIMADRA = {
    "small": dict(width=2048, heads=16, kv=4, dim=128, chunk=1024, q_rank=768, kv_rank=512, mem_heads=4, mem_dim=256, mem_vdim=512, ff=8192, layers=8, vocab=32000),
    "large": dict(width=4096, heads=32, kv=8, dim=128, chunk=2048, q_rank=1536, kv_rank=512, mem_heads=8, mem_dim=256, mem_vdim=512, ff=16384, layers=4, vocab=32000),
}
ARCHS = {"llama": LLAMA, "vebisun": VEBISUN, "fimadra": FIMADRA}
SINK = 4

# (N, K) of the products of the two Llama architectures, and two whose sizes fit no tile
PRODUCTS = [(5632, 2048), (2560, 2048), (2048, 5632), (32000, 2048), (6144, 4096), (4096, 4096), (28672, 4096), (14336, 4096), (4096, 14336), (1000, 1536), (3001, 2064)]


def listed():
    return [
        # the single operator of the smallest model, one row of f32 activations, weights as the unfused graph holds them
        dict(name="operator_f32_m1", kind="operator", m=1, n=5632, k=2048, dtype="f32", axis=1),
        # a prompt of odd length through one wide W8A8 product
        dict(name="w8a8_m777", kind="w8a8", m=777, n=14336, k=4096, dtype="bf16"),
        # one user at a small model: nothing but latency
        dict(name="step_tinyllama_b1", kind="step", arch="tinyllama", batch=1, context=192, dtype="f16", kv="16bit", host=True),
        # the serving step that the benchmark reports
        dict(name="step_8b_b32", kind="step", arch="llama3-8b", batch=32, context=2048, dtype="bf16", kv="16bit", host=False),
        # a few users with long odd contexts in the int8 cache
        dict(name="step_8b_b5_int8kv", kind="step", arch="llama3-8b", batch=5, context=3001, dtype="bf16", kv="int8", host=True),
        # two endless chats
        dict(name="stream_tinyllama_b2", kind="stream", arch="tinyllama", batch=2, window=1020, position=70001, dtype="bf16", kv="16bit"),
        # a long prompt, time to the first token
        dict(name="prompt_8b_2048", kind="request", family="llama", arch="llama3-8b", batch=1, prompt=2048, steps=0, dtype="bf16", kv="16bit"),
        # three short odd prompts and the first tokens of their answers
        dict(name="request_tinyllama_b3", kind="request", family="llama", arch="tinyllama", batch=3, prompt=333, steps=8, dtype="f16", kv="16bit"),
        # many small experts: one user, mostly decoding
        dict(name="request_vebisun_small", kind="request", family="vebisun", arch="small-experts", batch=1, prompt=500, steps=24, dtype="bf16", kv="16bit"),
        # few large experts: mostly prompts
        dict(name="request_vebisun_large", kind="request", family="vebisun", arch="large-experts", batch=4, prompt=505, steps=2, dtype="bf16", kv="16bit"),
        # recurrent and latent layers: a batch, mostly decoding
        dict(name="request_fimadra_small", kind="request", family="fimadra", arch="small", batch=8, prompt=130, steps=24, dtype="bf16", kv="16bit"),
        # recurrent and latent layers: one long prompt
        dict(name="prompt_fimadra_large", kind="request", family="fimadra", arch="large", batch=1, prompt=2048, steps=1, dtype="bf16", kv="16bit"),
    ]


def _log(rng, low, high):
    return min(high, max(low, int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))))


def draw(rng):
    kind = rng.choice(["operator", "w8a8", "step", "step", "stream", "request", "request", "request"])
    if kind == "operator":
        n, k = rng.choice(PRODUCTS)
        m = _log(rng, 1, 2048)
        axis = 1 if m == 1 and rng.random() < 0.4 else 0
        return dict(kind=kind, m=m, n=n, k=k, dtype=rng.choice(["bf16", "bf16", "f16", "f32"]) if m <= 32 else rng.choice(["bf16", "f16"]), axis=axis)
    if kind == "w8a8":
        n, k = rng.choice([p for p in PRODUCTS if p[1] % 16 == 0])
        return dict(kind=kind, m=_log(rng, 1, 2048), n=n, k=k, dtype="bf16")
    if kind == "step":
        arch = rng.choice(sorted(LLAMA))
        batch = _log(rng, 1, 32)
        return dict(kind=kind, arch=arch, batch=batch, context=_log(rng, 40, min(8192, 65536 // batch)), dtype="f16" if arch == "tinyllama" and rng.random() < 0.5 else "bf16",
                    kv=rng.choice(["16bit", "16bit", "int8"]), host=batch <= 8)
    if kind == "stream":
        window = _log(rng, 100, 4000)
        return dict(kind=kind, arch="tinyllama", batch=_log(rng, 1, 8), window=window, position=rng.randint(SINK + window, 200000), dtype="bf16",
                    kv=rng.choice(["16bit", "16bit", "int8"]))
    family = rng.choice(["llama", "vebisun", "fimadra"])
    arch = rng.choice(sorted(ARCHS[family]))
    batch = _log(rng, 1, 8)
    tokens, steps = (1536, 3) if arch == "llama3-8b" else (2048, 16)
    return dict(kind=kind, family=family, arch=arch, batch=batch, prompt=_log(rng, 20, tokens // batch), steps=rng.randint(0, steps), dtype="bf16",
                kv="int8" if family == "llama" and rng.random() < 0.25 else "16bit")


# ---- inputs ------------------------------------------------------------------------------------------------------------------------
def _gen(seed, stream=0):
    return torch.Generator(device="cuda").manual_seed(int(seed) * 1009 + stream)


def _int8_rows(shape, g):
    """Int8 rows as a per-row quantiser leaves normally distributed numbers."""
    return (torch.randn(shape, generator=g, device="cuda") * 32.0).round_().clamp_(-127, 127).to(torch.int8)


def _quantised(n, k, g, std):
    return _int8_rows((n, k), g), ((0.9 + 0.2 * torch.rand(n, generator=g, device="cuda")) * (std / 32.0)).bfloat16()


def _llama_weights(cfg, seed):
    """Checkpoint tensors by their usual names, quantised per row: weights like N(0, 0.02), those that write to the residual stream smaller by
    the root of their number, embedding rows of size one, so that the stream has the proportions of a trained model's."""
    g, out = _gen(seed), {}
    h, f, v, d = cfg["hidden_size"], cfg["intermediate_size"], cfg["vocab_size"], cfg["head_dim"]
    nq, nkv = cfg["num_attention_heads"] * d, cfg["num_key_value_heads"] * d
    shapes = {"model.embed_tokens.weight": (v, h), "lm_head.weight": (v, h)}
    for i in range(cfg["num_hidden_layers"]):
        p = f"model.layers.{i}."
        shapes.update({p + "self_attn.q_proj.weight": (nq, h), p + "self_attn.k_proj.weight": (nkv, h), p + "self_attn.v_proj.weight": (nkv, h),
                       p + "self_attn.o_proj.weight": (h, nq), p + "mlp.gate_proj.weight": (f, h), p + "mlp.up_proj.weight": (f, h), p + "mlp.down_proj.weight": (h, f)})
        for n in ("input_layernorm", "post_attention_layernorm"):
            out[p + n + ".weight"] = (1.0 + 0.1 * torch.randn(h, generator=g, device="cuda")).bfloat16()
    out["model.norm.weight"] = (1.0 + 0.1 * torch.randn(h, generator=g, device="cuda")).bfloat16()
    for n, (rows, cols) in shapes.items():
        std = 1.0 if "embed" in n else 0.02 / math.sqrt(2 * cfg["num_hidden_layers"]) if "o_proj" in n or "down_proj" in n else 0.02
        out[n], out[n + ".scale"] = _quantised(rows, cols, g, std)
    return out


def _context(case, cfg, seed, layer, which, rows):
    """Cached keys (which 0) or values (1) of one layer: [batch, kv heads, rows, head dim], and their scales with an int8 cache.  The
    spread is that of the projections' outputs, so a few rows stand out in the softmax, as in a trained model."""
    g = _gen(seed, 2 * layer + which + 1)
    shape = (case["batch"], cfg["num_key_value_heads"], rows, cfg["head_dim"])
    td = DTYPES[case["dtype"]]
    if case["kv"] == "int8":
        return _int8_rows(shape, g), ((0.9 + 0.2 * torch.rand(shape[:3], generator=g, device="cuda")) * (1.25 / 32)).to(td)
    return torch.empty(shape, dtype=td, device="cuda").normal_(0.0, 1.25, generator=g), None


def _tokens(vocab, seed, *shape):
    return torch.randint(0, vocab, shape, generator=torch.Generator().manual_seed(int(seed)))


def _vebisun_config(a):
    attn = dict(heads=a["heads"], kv_heads=a["kv"], dim=a["dim"], vdim=a["dim"], conv=4, scale=a["dim"] ** -0.5, softcap=30.0, mask=dict(size=a["window"]),
                rot=dict(base=5e5, dims=a["dim"] // 2, scaling=dict(factor=8.0, low=1.0, high=4.0, original=8192.0)))
    mlp = dict(kind="moe", expert=dict(ff=a["ff"]), router=dict(experts=a["experts"], top=a["top"], groups=dict(count=a["groups"], keep=a["keep"])))
    return dict(architecture="Vebisun", width=a["width"], vocab=a["vocab"], layers=[dict(type="attention", mixer=attn, mlp=mlp)] * a["layers"],
                embedding=dict(scale=1.0), residual_mult=0.5, norm=dict(eps=1e-5))


def _fimadra_config(a):
    h, d, mlp = a["heads"], a["dim"], dict(kind="dense", ff=a["ff"])
    latent = dict(type="latent_attention", mlp=mlp, mixer=dict(heads=h, dim=d, vdim=d, scale=d ** -0.5, q_rank=a["q_rank"], kv_rank=a["kv_rank"]))
    attn = dict(type="attention", mlp=mlp, mixer=dict(heads=h, kv_heads=a["kv"], dim=d, vdim=d, scale=d ** -0.5, mask=dict(size=a["chunk"]), rot=dict(base=1e6, dims=d)))
    mem = dict(type="mlstm", mlp=None, mixer=dict(heads=a["mem_heads"], dim=a["mem_dim"], vdim=a["mem_vdim"], gate_cap=15.0))
    return dict(architecture="Fimadra", width=a["width"], vocab=a["vocab"], layers=([latent, attn, mem, mem] * a["layers"])[:a["layers"]], norm=dict(eps=1e-6), logit_scale=0.5)


def _routed_part(router, r, vocab, size, g):
    """What the embedding rows hold of the directions of the experts that a token goes to: a trained router is decided, not a toss-up
    among random scores."""
    groups = r["groups"]
    kept = torch.rand(vocab, groups["count"], generator=g, device="cuda").topk(groups["keep"], -1).indices
    score = torch.rand(vocab, groups["count"], r["experts"] // groups["count"], generator=g, device="cuda")
    score += torch.zeros_like(score[..., 0]).scatter_(1, kept, 1.0)[..., None]
    chosen = score.view(vocab, -1).topk(r["top"], -1).indices
    share = torch.zeros(vocab, r["experts"], device="cuda").scatter_(1, chosen, size)
    return (share @ torch.nn.functional.normalize(router.float(), dim=-1)).bfloat16()


def _block_weights(family, cfg, seed):
    g, w, out = _gen(seed), cfg["width"], {}

    def mat(name, *shape, std=0.02):
        out[name] = torch.empty(*shape, device="cuda", dtype=torch.bfloat16).normal_(0.0, std, generator=g)

    def vec(name, n, mean):
        out[name] = (mean + 0.1 * torch.randn(n, generator=g, device="cuda")).bfloat16()

    def norm(name):
        vec(name, w, 1.0)
        if family == "vebisun":
            vec(name + ".b", w, 0.0)

    mat("embed", cfg["vocab"], w, std=2.0 if family == "vebisun" else 0.02)
    mat("head", cfg["vocab"], w)
    norm("final.norm")
    for i, entry in enumerate(cfg["layers"]):
        p, m, mlp = f"l{i}.", entry["mixer"], entry["mlp"]
        h, d, e = m["heads"], m["dim"], m["vdim"]
        for n in ("norm1", "norm1b") if family == "vebisun" else ("norm1",):
            norm(p + n)
        if entry["type"] == "attention":
            for n, rows in (("q", h * d), ("k", m["kv_heads"] * d), ("v", m["kv_heads"] * e)):
                mat(p + "mix." + n, rows, w)
                if m.get("conv"):  # the token itself first, its predecessors less
                    mat(p + f"mix.{n}.conv", rows, m["conv"], std=0.2)
                    out[p + f"mix.{n}.conv"][:, -1] += 1.0
        elif entry["type"] == "latent_attention":
            mat(p + "mix.dq", m["q_rank"], w)
            mat(p + "mix.dkv", m["kv_rank"], w)
            vec(p + "mix.dq.norm", m["q_rank"], 1.0)
            vec(p + "mix.dkv.norm", m["kv_rank"], 1.0)
            mat(p + "mix.uq", h * d, m["q_rank"], std=0.04)
            mat(p + "mix.uk", h * d, m["kv_rank"], std=0.04)
            mat(p + "mix.uv", h * e, m["kv_rank"], std=0.04)
        else:
            for n, rows in (("q", h * d), ("k", h * d), ("v", h * e), ("g", h * e), ("i", h), ("f", h)):
                mat(p + "mix." + n, rows, w)
            vec(p + "mix.i.b", h, 0.0)
            vec(p + "mix.f.b", h, 4.0)
            vec(p + "mix.norm", h * e, 1.0)
        mat(p + "mix.o", w, h * e)
        if mlp:
            for n in ("norm2", "norm2b") if family == "vebisun" else ("norm2",):
                norm(p + n)
            if mlp["kind"] == "moe":
                r, ff = mlp["router"], mlp["expert"]["ff"]
                mat(p + "mlp.router", r["experts"], w, std=1.5 * w ** -0.5)
                out["embed"] += _routed_part(out[p + "mlp.router"], r, cfg["vocab"], 16.0, g)
                for j in range(r["experts"]):
                    for n, shape in (("gate", (ff, w)), ("up", (ff, w)), ("down", (w, ff))):
                        mat(f"{p}mlp.e{j}.{n}", *shape)
            else:
                mat(p + "mlp.up", mlp["ff"], w)
                mat(p + "mlp.down", w, mlp["ff"])
    return out


def _operands(case, seed):
    g, td = _gen(seed), DTYPES[case["dtype"]]
    m, n, k = case["m"], case["n"], case["k"]
    act = torch.randn(m, k, generator=g, device="cuda").to(td)
    w, scale = _quantised(n, k, g, 0.02)
    return act, w, scale.to(td)


_STREAM = []


def _stream():
    """The stream of the program's device-resident steps."""
    if not _STREAM:
        _STREAM.append(torch.cuda.Stream())
    return _STREAM[0]


def _chunk(case):
    return min(case["prompt"], max(64, 2048 // case["batch"]))


def prepare(case, seed):
    kind = case["kind"]
    if kind in ("operator", "w8a8"):
        act, w, scale = _operands(case, seed)
        if kind == "operator":
            return dict(case=case, act=act, w=w.t().contiguous() if case["axis"] == 1 else w, scale=scale)
        return dict(case=case, act=act, w=w, scale=scale)
    if kind == "request":
        family = case["family"]
        cfg = ARCHS[family][case["arch"]]
        total, vocab = case["prompt"] + case["steps"], cfg.get("vocab_size") or cfg["vocab"]
        kw = dict(dtype=case["dtype"], max_seq_len=-(-(total + 1) // 256) * 256, batch=case["batch"], output="logits", max_prefill=_chunk(case))
        if family == "llama":
            model = DecoderModel(cfg, _llama_weights(cfg, seed), kv_int8=case["kv"] == "int8", **kw)
        else:
            cfg = (_vebisun_config if family == "vebisun" else _fimadra_config)(cfg)
            model = (vebisun if family == "vebisun" else fimadra).build(cfg, _block_weights(family, cfg, seed), **kw)
        return dict(case=case, model=model, tokens=_tokens(vocab, seed, case["batch"], total), logits=DTYPES[case["dtype"]] if family == "llama" else torch.float32)
    cfg = LLAMA[case["arch"]]
    streaming = (SINK, case["window"]) if kind == "stream" else None
    rows = SINK + case["window"] if kind == "stream" else case["context"]
    model = DecoderModel(cfg, _llama_weights(cfg, seed), dtype=case["dtype"], batch=case["batch"], output="logits", kv_int8=case["kv"] == "int8", streaming=streaming,
                         max_seq_len=-(-rows // 8) * 8 if streaming else -(-(rows + 1) // 256) * 256)
    for i in range(cfg["num_hidden_layers"]):
        for which, (cache, scales) in enumerate(((model.k_cache, model.k_scale), (model.v_cache, model.v_scale))):
            t, s = _context(case, cfg, seed, i, which, rows)
            cache[i][:, :, :rows].copy_(t)
            if s is not None:
                scales[i][:, :, :rows].copy_(s)
    tokens = _tokens(cfg["vocab_size"], seed, case["batch"])
    state = dict(case=case, model=model, tokens=tokens)
    if not case.get("host", True):
        state.update(tokens=tokens.cuda(), out=torch.empty(case["batch"], cfg["vocab_size"], dtype=DTYPES[case["dtype"]], device="cuda"))
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "operator":
        return ops.dequant_matmul(state["act"], state["w"], state["scale"], axis=case["axis"])
    if kind == "w8a8":
        y, y_scale, _ = ops.dynamic_quantize_linear(state["act"])
        return ops.quantized_matmul(y, y_scale, state["w"], state["scale"])
    model, tokens = state["model"], state["tokens"]
    if kind == "stream":
        return model.stream(tokens, case["position"])
    if kind == "step":
        if case["host"]:
            return model.step(tokens, case["context"])
        model.step_device(tokens, case["context"], state["out"], _stream().cuda_stream)
        return state["out"]
    prompt, chunk, logits = case["prompt"], _chunk(case), torch.empty(case["steps"] + 1, case["batch"], model.vocab, dtype=state["logits"])
    for p in range(0, prompt, chunk):
        out = model.prefill(tokens[:, p:min(p + chunk, prompt)], p)
    logits[0] = out
    for i in range(case["steps"]):
        logits[i + 1] = model.step(tokens[:, prompt + i], prompt + i)
    if not _returns_state(case):
        return dict(logits=logits)
    return dict(logits=logits, state=_state_tensors(case, model))


def _returns_state(case):
    """Whether the caches can be compared value by value: an int8 row may round either way, and a routed token near a tie may go to
    another expert altogether.  They then show in the logits of the later steps only."""
    return case["kv"] != "int8" and case["family"] != "vebisun"


def _state_tensors(case, model):
    """The caches that a pass has filled: of at most the last 16 layers (what came before them shows in theirs)."""
    if case["family"] == "llama":
        return [t for kv in list(zip(model.k_cache, model.v_cache))[-16:] for t in kv]
    return [t for layer in model.run_states for t in layer if t is not None]


# ---- what a pass cannot do without -------------------------------------------------------------------------------------------------
def _llama_numbers(cfg):
    h, f, d = cfg["hidden_size"], cfg["intermediate_size"], cfg["head_dim"]
    nq, nkv = cfg["num_attention_heads"] * d, cfg["num_key_value_heads"] * d
    return cfg["num_hidden_layers"] * ((nq + 2 * nkv) * h + h * nq + 3 * f * h), cfg["vocab_size"] * h


def _tokens_cost(case, tokens, first, last):
    """(weight numbers read, flops without the head, bytes of cache read) of a pass over ``tokens`` rows, positions first .. last - 1 of each
    sequence."""
    family, b = case.get("family", "llama"), case["batch"]
    if family == "llama":
        cfg = LLAMA[case["arch"]]
        body, _ = _llama_numbers(cfg)
        pairs = sum(min(p + 1, case.get("window", 10 ** 9) + SINK) for p in range(first, last))
        row = 2 * cfg["num_key_value_heads"] * (cfg["head_dim"] * (1 if case["kv"] == "int8" else 2) + (2 if case["kv"] == "int8" else 0))
        seen = min(last, case.get("window", 10 ** 9) + SINK)
        return (body, 2.0 * tokens * body + 4.0 * b * pairs * cfg["num_hidden_layers"] * cfg["num_attention_heads"] * cfg["head_dim"],
                b * seen * row * cfg["num_hidden_layers"])
    a = ARCHS[family][case["arch"]]
    w, h, d = a["width"], a["heads"], a["dim"]
    if family == "vebisun":
        fixed = (h + 2 * a["kv"]) * d * w + w * h * d + a["experts"] * w
        used = a["experts"] * (1.0 - (1.0 - a["top"] / a["experts"]) ** tokens)
        pairs = sum(min(p + 1, a["window"]) for p in range(first, last))
        layer = (fixed + used * 3 * a["ff"] * w, 2.0 * tokens * (fixed + a["top"] * 3 * a["ff"] * w) + 4.0 * b * pairs * h * d, 4.0 * b * min(last, a["window"] + last - first) * a["kv"] * d)
        return tuple(a["layers"] * v for v in layer)
    total = [0.0, 0.0, 0.0]
    ff = 2 * a["ff"] * w
    for i in range(a["layers"]):
        if i % 4 == 0:
            n = (a["q_rank"] + a["kv_rank"]) * w + h * d * (a["q_rank"] + 2 * a["kv_rank"]) + w * h * d + ff
            pairs, cache = sum(range(first + 1, last + 1)), 2.0 * b * last * a["kv_rank"]
            flops = 2.0 * tokens * n + 4.0 * b * pairs * h * d
        elif i % 4 == 1:
            n = (h + 2 * a["kv"]) * d * w + w * h * d + ff
            pairs, cache = sum(p % a["chunk"] + 1 for p in range(first, last)), 4.0 * b * min(last, a["chunk"]) * a["kv"] * d
            flops = 2.0 * tokens * n + 4.0 * b * pairs * h * d
        else:
            cells = a["mem_heads"] * a["mem_dim"] * a["mem_vdim"]
            n = a["mem_heads"] * (2 * a["mem_dim"] + 2 * a["mem_vdim"] + 2) * w + w * a["mem_heads"] * a["mem_vdim"]
            flops, cache = 2.0 * tokens * n + 4.0 * tokens * cells, 8.0 * b * cells
        for j, v in enumerate((n, flops, cache)):
            total[j] += v
    return tuple(total)


def work(case):
    kind = case["kind"]
    if kind in ("operator", "w8a8"):
        m, n, k, e = case["m"], case["n"], case["k"], torch.empty(0, dtype=DTYPES[case["dtype"]]).element_size()
        return dict(bytes=n * k + e * (n + m * k + m * n), flops=2.0 * m * n * k)
    family, b = case.get("family", "llama"), case["batch"]
    if family == "llama":
        head, size = _llama_numbers(LLAMA[case["arch"]])[1], 1
        vocab = LLAMA[case["arch"]]["vocab_size"]
    else:
        a = ARCHS[family][case["arch"]]
        head, size, vocab = a["vocab"] * a["width"], 2, a["vocab"]
    out = b * vocab * (4 if family != "llama" else 2)
    if kind == "request":
        spans = [(0, case["prompt"])] + [(p, p + 1) for p in range(case["prompt"], case["prompt"] + case["steps"])]
    elif kind == "step":
        spans = [(case["context"], case["context"] + 1)]
    else:
        spans = [(case["position"], case["position"] + 1)]
    total = dict(bytes=0.0, flops=0.0)
    for first, last in spans:
        weights, flops, cache = _tokens_cost(case, b * (last - first), first, last)
        total["bytes"] += size * (weights + head) + cache + out
        total["flops"] += flops + 2.0 * b * head
    return total


def tolerance(case):
    kind = case["kind"]
    if kind == "operator":
        return {"rel": 1e-5} if case["dtype"] == "f32" else {"rel": 1e-2}
    if kind == "w8a8":  # whole-number sums: only the last roundings
        return {"rel": 1e-2}
    # every stored row is rounded, and 22 or 32 layers carry it on; with the other kernels of this library that the options choose
    # (another order of sums in attention) f16 models are 0.0013 apart, bf16 ones 0.022 (32 layers), 0.009 (Fimadra) and 0.0035 (Vebisun,
    # whose residual stream is f32 and mostly its embedding)
    if case.get("family") == "vebisun":
        return {"rel": 0.015, "max": 0.1}
    return {"rel": 0.006, "max": 0.05} if case["dtype"] == "f16" else {"rel": 0.03, "max": 0.5}


# ---- the same in 64 bits -----------------------------------------------------------------------------------------------------------
def exact(case, seed):
    kind = case["kind"]
    with torch.no_grad():
        if kind == "operator":
            act, w, scale = _operands(case, seed)
            return (act.double() @ w.double().t()) * scale.double()
        if kind == "w8a8":
            act, w, scale = _operands(case, seed)
            x = act.double()
            step = (x.abs().amax(1, keepdim=True) / 127.0).float().double()
            y = (x / step).round().clamp(-128, 127)
            return (y * step) @ w.double().t() * scale.double()
        if case.get("family", "llama") == "llama":
            return _exact_llama(case, seed)
        return _exact_block(case, seed)


def _attend(q, k, v, scale, allowed=None, softcap=0.0):
    """q [B, Hq, S, D], k / v [B, G, L, .], allowed [S, L] -> [B, S, Hq * E]."""
    out = []
    rep = q.shape[1] // k.shape[1]
    for b in range(q.shape[0]):
        s = q[b].reshape(k.shape[1], -1, q.shape[3]) @ k[b].transpose(1, 2) * scale  # [G, rep * S, L]
        if softcap:
            s = softcap * torch.tanh(s / softcap)
        if allowed is not None:
            s = s.masked_fill(~allowed.repeat(rep, 1), -math.inf)
        o = torch.softmax(s, -1) @ v[b]
        out.append(o.reshape(q.shape[1], q.shape[2], -1).transpose(0, 1).reshape(q.shape[2], -1))
    return torch.stack(out)


def _heads(x, n):
    return x.view(x.shape[0], x.shape[1], n, -1).transpose(1, 2)


def _rotate_halves(x, cos, sin):
    half = x.shape[-1] // 2
    return x * cos + torch.cat([-x[..., half:], x[..., :half]], -1) * sin


def _llama_tables(cfg, positions, dtype):
    """cos and sin at these positions as the tables hold them: bf16 cut off, f16 rounded."""
    d = cfg["head_dim"]
    freqs = np.array([1.0 / float(np.float32(cfg["rope_theta"])) ** (2.0 * i / d) for i in range(d // 2)])
    angles = np.asarray(positions, dtype=np.float64)[:, None] * np.concatenate([freqs, freqs])[None, :]
    out = []
    for t in (np.cos(angles), np.sin(angles)):
        t = t.astype(np.float32)
        t = (t.view(np.uint32) & np.uint32(0xFFFF0000)).view(np.float32) if dtype == "bf16" else t.astype(np.float16)
        out.append(torch.from_numpy(t.astype(np.float64)).cuda())
    return out


def _int8_round_trip(x):
    step = x.abs().amax(-1, keepdim=True) / 127.0
    return (x / step).round().clamp(-128, 127) * step


def _exact_llama(case, seed):
    cfg, kind, kv8 = LLAMA[case["arch"]], case["kind"], case["kv"] == "int8"
    w = _llama_weights(cfg, seed)
    td = DTYPES[case["dtype"]]
    hq, hkv, d, eps = cfg["num_attention_heads"], cfg["num_key_value_heads"], cfg["head_dim"], cfg["rms_norm_eps"]
    b = case["batch"]

    def linear(x, name):
        return (x @ w[name].double().t()) * w[name + ".scale"].to(td).double()

    def norm(x, name):
        return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps) * w[name].to(td).double()

    if kind == "request":
        total = case["prompt"] + case["steps"]
        tokens, positions = _tokens(cfg["vocab_size"], seed, b, total).cuda(), np.arange(total)
        allowed = torch.ones(total, total, dtype=torch.bool, device="cuda").tril()
    else:
        tokens, allowed = _tokens(cfg["vocab_size"], seed, b).cuda()[:, None], None
        positions = [case["context"] if kind == "step" else SINK + case["window"] - 1]
    cos, sin = _llama_tables(cfg, positions, case["dtype"])
    if kind == "stream":  # slots by age: the sink, then the ring from the oldest entry on; the new token takes the oldest one's place
        window, slots = case["window"], SINK + case["window"]
        new = SINK + (case["position"] - SINK) % window
        order = list(range(SINK)) + [SINK + (new - SINK + 1 + i) % window for i in range(window)]
        ring_cos, ring_sin = _llama_tables(cfg, np.arange(slots), case["dtype"])
    caches = []
    name = "model.embed_tokens.weight"
    x = w[name][tokens].double() * w[name + ".scale"].to(td).double()[tokens][..., None]
    for i in range(cfg["num_hidden_layers"]):
        p = f"model.layers.{i}."
        n = norm(x, p + "input_layernorm.weight")
        q, k, v = (_heads(linear(n, p + f"self_attn.{c}_proj.weight"), heads) for c, heads in (("q", hq), ("k", hkv), ("v", hkv)))
        q = _rotate_halves(q, cos, sin)
        if kind != "stream":
            k = _rotate_halves(k, cos, sin)
        if kv8:
            k, v = _int8_round_trip(k), _int8_round_trip(v)
        if kind != "request":
            past = []
            for which in (0, 1):
                t, s = _context(case, cfg, seed, i, which, slots if kind == "stream" else case["context"])
                past.append(t.double() if s is None else t.double() * s.double()[..., None])
            if kind == "step":
                k, v = torch.cat([past[0], k], 2), torch.cat([past[1], v], 2)
            else:
                past[0][:, :, new], past[1][:, :, new] = k[:, :, 0], v[:, :, 0]
                k, v = _rotate_halves(past[0][:, :, order], ring_cos, ring_sin), past[1][:, :, order]
        else:
            caches.append((k, v))
        x = x + linear(_attend(q, k, v, d ** -0.5, allowed), p + "self_attn.o_proj.weight")
        n = norm(x, p + "post_attention_layernorm.weight")
        x = x + linear(torch.nn.functional.silu(linear(n, p + "mlp.gate_proj.weight")) * linear(n, p + "mlp.up_proj.weight"), p + "mlp.down_proj.weight")
    at = x[:, case["prompt"] - 1:] if kind == "request" else x
    logits = linear(norm(at, "model.norm.weight"), "lm_head.weight")
    if kind != "request":
        return logits[:, 0]
    if not _returns_state(case):
        return dict(logits=logits.transpose(0, 1))
    rows = -(-(total + 1) // 256) * 256
    state = []
    for kv in caches[-16:]:
        for t in kv:
            c = torch.zeros(b, hkv, rows, d, dtype=torch.float64, device="cuda")
            c[:, :, :total] = t
            state.append(c)
    return dict(logits=logits.transpose(0, 1), state=state)


def _ring(t, rows):
    """Position p of t [B, heads, T, .] in row p % rows; the later position stays."""
    total = t.shape[2]
    out = torch.zeros(*t.shape[:2], rows, t.shape[3], dtype=t.dtype, device=t.device)
    last = torch.arange(max(0, total - rows), total, device=t.device)
    out[:, :, last % rows] = t[:, :, last]
    return out


def _rms(x, eps):
    return x * torch.rsqrt((x * x).mean(-1, keepdim=True) + eps)


def _exact_block(case, seed):
    family, b = case["family"], case["batch"]
    cfg = (_vebisun_config if family == "vebisun" else _fimadra_config)(ARCHS[family][case["arch"]])
    w, eps = _block_weights(family, cfg, seed), cfg["norm"]["eps"]
    total = case["prompt"] + case["steps"]
    tokens = _tokens(cfg["vocab"], seed, b, total).cuda()
    max_seq, rewind, at = -(-(total + 1) // 256) * 256, 32, torch.arange(total, device="cuda")

    def linear(x, name):
        return x @ w[name].double().t()

    def norm(x, name):
        if family == "fimadra":
            return _rms(x, eps) * w[name].double()
        return torch.nn.functional.layer_norm(x, x.shape[-1:], w[name].double(), w[name + ".b"].double(), eps)

    def ring_rows(reach):
        return -(-min(max_seq, reach - 1 + _chunk(case) + rewind) // 128) * 128

    def rotate(x, base, dims, halves, scaling=None):
        f = base ** (-2.0 * np.arange(dims // 2, dtype=np.float64) / dims)
        if scaling:
            turns = scaling["original"] * f / (2.0 * math.pi)
            share = np.clip((turns - scaling["low"]) / (scaling["high"] - scaling["low"]), 0.0, 1.0)
            f = f * (share + (1.0 - share) / scaling["factor"])
        angle = at.double()[:, None] * torch.from_numpy(f).cuda()
        c, s, y = angle.cos(), angle.sin(), x.clone()
        u, v = (x[..., :dims // 2], x[..., dims // 2:dims]) if halves else (x[..., 0:dims:2], x[..., 1:dims:2])
        a, o = u * c - v * s, v * c + u * s
        if halves:
            y[..., :dims // 2], y[..., dims // 2:dims] = a, o
        else:
            y[..., 0:dims:2], y[..., 1:dims:2] = a, o
        return y

    state = []

    def attention(x, p, m):
        raw = [linear(x, p + "mix." + n) for n in "qkv"]
        if m.get("conv"):
            rows = m["conv"] + rewind
            state_conv = _ring(torch.cat(raw, -1)[:, None], rows)[:, 0]
            mixed = []
            for n, t in zip("qkv", raw):
                taps, y = w[p + f"mix.{n}.conv"].double(), torch.zeros_like(t)
                for j in range(m["conv"]):
                    lag = m["conv"] - 1 - j
                    if lag < total:
                        y[:, lag:] += taps[:, j] * t[:, :total - lag]
                mixed.append(y)
            raw = mixed
        q, k, v = _heads(raw[0], m["heads"]), _heads(raw[1], m["kv_heads"]), _heads(raw[2], m["kv_heads"])
        rot, size = m["rot"], m["mask"]["size"]
        q, k = (rotate(t, rot["base"], rot["dims"], family == "fimadra", rot.get("scaling")) for t in (q, k))
        back = at[:, None] - at[None, :]
        if family == "fimadra":
            q, k = _rms(q, eps), _rms(k, eps)
            allowed = (back >= 0) & (at[:, None] // size == at[None, :] // size)
        else:
            allowed = (back >= 0) & (back < size)
        state.extend([_ring(k, ring_rows(size)), _ring(v, ring_rows(size))] + ([state_conv] if m.get("conv") else []))
        return linear(_attend(q, k, v, m["scale"], allowed, m.get("softcap") or 0.0), p + "mix.o")

    def latent(x, p, m):
        cq, c = (_rms(linear(x, p + "mix." + n), eps) * w[p + f"mix.{n}.norm"].double() for n in ("dq", "dkv"))
        q, k, v = _heads(linear(cq, p + "mix.uq"), m["heads"]), _heads(linear(c, p + "mix.uk"), m["heads"]), _heads(linear(c, p + "mix.uv"), m["heads"])
        state.append(_ring(c[:, None], -(-max_seq // 128) * 128)[:, 0])
        return linear(_attend(q, k, v, m["scale"], at[:, None] >= at[None, :]), p + "mix.o")

    def memory(x, p, m):
        h, cap = m["heads"], m["gate_cap"]
        q, k, v, z = (linear(x, p + "mix." + n) for n in "qkvg")
        q, k, v = _heads(q, h) * m["dim"] ** -0.5, _heads(k, h), _heads(v, h)
        take, keep = (cap * torch.tanh((linear(x, p + "mix." + n) + w[p + f"mix.{n}.b"].double()) / cap) for n in "if")
        take, run = take.transpose(1, 2), torch.nn.functional.logsigmoid(keep).cumsum(1).transpose(1, 2)  # [B, H, T]
        out = []
        last = []
        for i in range(b):  # weight of token s at t: exp(run_t - run_s + take_s - top_t), with the empty memory's own at exp(run_t - top_t)
            d = (run[i, :, :, None] - run[i, :, None, :] + take[i, :, None, :]).masked_fill(at[:, None] < at[None, :], -math.inf)
            top = torch.maximum(d.amax(-1), run[i])
            d = (d - top[..., None]).exp_()
            s = (q[i] @ k[i].transpose(1, 2)).mul_(d)
            out.append((s @ v[i]) / (torch.maximum(s.sum(-1).abs(), (-top).exp()) + 1e-6)[..., None])
            share = d[:, -1, :, None] * k[i]
            last.append((share.transpose(1, 2) @ v[i], share.sum(1), top[:, -1]))
        state.extend(torch.stack(t) for t in zip(*last))
        o = _rms(torch.stack(out), eps).transpose(1, 2).reshape(b, total, -1) * w[p + "mix.norm"].double()
        return linear(o * torch.sigmoid(z), p + "mix.o")

    def experts(x, p, mlp):
        r, y = mlp["router"], torch.zeros_like(x).reshape(-1, x.shape[-1])
        flat = x.reshape(-1, x.shape[-1])
        score = torch.softmax(linear(flat, p + "mlp.router"), -1)
        by_group = score.view(-1, r["groups"]["count"], r["experts"] // r["groups"]["count"])
        kept = by_group.amax(-1).topk(r["groups"]["keep"], -1).indices
        mask = torch.zeros(by_group.shape[:2], dtype=torch.bool, device="cuda").scatter_(1, kept, True)
        chosen = by_group.masked_fill(~mask[..., None], -1.0).view_as(score).topk(r["top"], -1).indices
        for j in range(r["experts"]):
            rows = (chosen == j).any(-1).nonzero()[:, 0]
            if rows.numel():
                t, e = flat[rows], f"{p}mlp.e{j}."
                y.index_add_(0, rows, score[rows, j, None] * linear(torch.nn.functional.silu(linear(t, e + "gate")) * linear(t, e + "up"), e + "down"))
        return y.view_as(x)

    mixers = {"attention": attention, "latent_attention": latent, "mlstm": memory}
    x = w["embed"][tokens].double()
    for i, entry in enumerate(cfg["layers"]):
        p = f"l{i}."
        y = mixers[entry["type"]](norm(x, p + "norm1"), p, entry["mixer"])
        x = x + (cfg["residual_mult"] * norm(y, p + "norm1b") if family == "vebisun" else y)
        if entry["mlp"]:
            n = norm(x, p + "norm2")
            if family == "vebisun":
                x = x + cfg["residual_mult"] * norm(experts(n, p, entry["mlp"]), p + "norm2b")
            else:
                x = x + linear(torch.relu(linear(n, p + "mlp.up")).square(), p + "mlp.down")
    logits = linear(norm(x[:, case["prompt"] - 1:], "final.norm"), "head") * cfg.get("logit_scale", 1.0)
    return dict(logits=logits.transpose(0, 1), state=state) if _returns_state(case) else dict(logits=logits.transpose(0, 1))
