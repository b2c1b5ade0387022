"""Forms that one operator is dispatched to, on both sides of each rule and at the edges of their tiles: integer sums are exact, so forms of
the int8 products agree to the last bit; the others are compared with float64."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

from my_nn_engine_b200 import ffi, ops  # noqa: E402
from oracle import ref_ops as R  # noqa: E402
from oracle import ref_vebisun as V  # noqa: E402

DT = {"bf16": torch.bfloat16, "f16": torch.float16, "f32": torch.float32}


def gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def randn(g, *shape):
    return torch.randn(*shape, generator=g, device="cuda")


def int8(g, *shape):
    return torch.randint(-127, 128, shape, generator=g, device="cuda", dtype=torch.int32).to(torch.int8)


def scales(g, n, dt):
    return (0.002 + 0.018 * torch.rand(n, generator=g, device="cuda")).to(dt)


def oracle_steps(cfg, state, dt, batch, rows, **options):
    """step(pos, tokens, caches) -> logits of the CPU oracle over given caches (torch tensors by attribute name, of the first layer), and the oracle."""
    from oracle.ref_model import LlamaConfig, OracleLlama
    weights = {n: t.cpu().numpy() if t.dtype == torch.int8 else R.store_round(t.float().cpu().numpy(), dt) for n, t in state.items()}
    oracle = OracleLlama(LlamaConfig.from_hf(cfg), weights, dt, rows, batch, c_attention="streaming" not in options, **options)

    def step(pos, tokens, caches):
        for name, t in caches.items():
            getattr(oracle, name)[0] = t.cpu().numpy() if t.dtype == torch.int8 else t.float().cpu().numpy()
        oracle.past_len = pos
        oracle.decode_step(tokens)
        return torch.from_numpy(oracle.last_logits).double()

    return step, oracle


# a layer and the head store about a dozen roundings of half an ulp (2^-9, 2^-12) on the way from the attention to the logits, which add up like a random walk
LAYER = {"bf16": 2.0 ** -6, "f16": 2.0 ** -9}


# ---- DequantMatMul of a few rows: up to five go to the lean kernel, eight to the tcgen05 one ----
@pytest.mark.parametrize("dt", ["bf16", "f16", "f32"])
@pytest.mark.parametrize("n,k", [(1, 16), (130, 1040), (2561, 2048), (2100, 4096), (700, 4112), (5000, 6144), (40001, 512), (9000, 4096)])
def test_lean_product_equals_the_tensor_core_product(dt, n, k):
    g = gen(n + k)
    w, s, act = int8(g, n, k), scales(g, n, DT[dt]), randn(g, 8, k).to(DT[dt])
    act[2] = 0
    res = randn(g, 8, n).to(DT[dt])
    want, want_res = ops.dequant_matmul(act, w, s), ops.dequant_matmul_residual(act, w, s, res)
    for m in (1, 2, 3, 4, 5):
        assert torch.equal(ops.dequant_matmul(act[:m], w, s), want[:m])
        assert torch.equal(ops.dequant_matmul_residual(act[:m], w, s, res[:m]), want_res[:m])
    for m in (1, 3, 8):
        shifted = torch.empty(m * k + 1, dtype=DT[dt], device="cuda")[1:].view(m, k)  # rows that no wider load may touch
        shifted.copy_(act[:m])
        assert torch.equal(ops.dequant_matmul(shifted, w, s), want[:m])
    act[1, k // 2] = float("inf")  # spoils its own row alone
    got = ops.dequant_matmul(act[:4], w, s)
    assert torch.isnan(got[1]).all() and torch.equal(got[[0, 2, 3]], want[[0, 2, 3]])


@pytest.mark.parametrize("dt", ["bf16", "f16"])
@pytest.mark.parametrize("hidden,ffn", [(256, 704), (512, 1040), (384, 512)])
def test_small_batches_step_like_a_large_one(dt, hidden, ffn):
    """A first token attends to itself alone, so a step of one to five sequences (lean products, limbs of the
    attention's rows made inside) and of eight (tcgen05 products) have to agree to the last bit."""
    from my_nn_engine_b200.decoder import DecoderModel
    from my_nn_engine_b200.quantize import random_llama_state
    cfg = dict(hidden_size=hidden, num_hidden_layers=2, num_attention_heads=hidden // 64, num_key_value_heads=2, head_dim=64, intermediate_size=ffn, vocab_size=500,
               rms_norm_eps=1e-5, rope_theta=1e4)
    state, tokens, rows = random_llama_state(cfg, seed=3), np.arange(8) * 61 % 500, {}
    for batch in (1, 2, 3, 5, 8):
        model = DecoderModel(cfg, state, dtype=dt, max_seq_len=32, batch=batch)
        rows[batch] = model.step(tokens[:batch], 0).clone()
        model.close()
    for batch in (1, 2, 3, 5):
        assert torch.equal(rows[batch], rows[8][:batch])


# gate/up products with the SiLU product in their finish: more than one pass over the partial sums, last shares of a few outputs, each number of blocks along K
@pytest.mark.parametrize("dt", ["bf16", "f16", "f32"])
@pytest.mark.parametrize("hidden,ffn", [(128, 9104), (1152, 1136), (2112, 304), (4160, 80)])
def test_gated_products_step_like_a_large_batch(dt, hidden, ffn):
    from my_nn_engine_b200.decoder import DecoderModel
    from my_nn_engine_b200.quantize import random_llama_state
    cfg = dict(hidden_size=hidden, num_hidden_layers=1, num_attention_heads=2, num_key_value_heads=1, head_dim=64, intermediate_size=ffn, vocab_size=300,
               rms_norm_eps=1e-5, rope_theta=1e4)
    state, tokens, rows = random_llama_state(cfg, seed=5), np.arange(8) * 37 % 300, {}
    for batch in (1, 2, 3, 4, 5, 8):
        model = DecoderModel(cfg, state, dtype=dt, max_seq_len=32, batch=batch)
        rows[batch] = model.step(tokens[:batch], 0).clone()
        model.close()
    for batch in (1, 2, 3, 4, 5):
        assert torch.equal(rows[batch], rows[8][:batch])


# ---- products of many int8 rows: tile widths, ragged last tiles ----
@pytest.mark.parametrize("m,n,k", [(257, 3001, 1040), (520, 128, 2064), (777, 14336, 256), (2047, 640, 512), (1500, 5632, 128), (40, 130, 16)])
def test_w8a8_product_is_exact(m, n, k):
    g = gen(m)
    a, w, sa, sw = int8(g, m, k), int8(g, n, k), scales(g, m, torch.bfloat16), scales(g, n, torch.bfloat16)
    want = ((a.double() @ w.double().t()).float() * sa.float()[:, None] * sw.float()).bfloat16()
    assert torch.equal(ops.quantized_matmul(a, sa, w, sw), want)


# a pair of CTAs owns 256 weight rows and up to 256 int8 rows: second CTA without rows, with one, tiles of 32 columns and one more, rings of six to nine stages
@pytest.mark.parametrize("m,n,k", [(33, 1, 16), (32, 128, 144), (95, 129, 1152), (97, 257, 1168), (256, 385, 784), (288, 19200, 128), (1025, 512, 896)])
def test_int8_products_of_cta_pairs_are_exact(m, n, k):
    g = gen(m + n)
    a, w, sa, sw = int8(g, m, k), int8(g, n, k), scales(g, m, torch.bfloat16), scales(g, n, torch.bfloat16)
    exact = a.double() @ w.double().t()
    assert torch.equal(ops.quantized_matmul(a, sa, w, sw), (exact.float() * sa.float()[:, None] * sw.float()).bfloat16())
    if m > 32:  # whole numbers up to 127 are their own limbs, so these sums are exact too; the residual is added behind a rounding of its own
        res = randn(g, m, n).bfloat16()
        want = (exact.float() * sw.float()).bfloat16()
        assert torch.equal(ops.dequant_matmul(a.bfloat16(), w, sw), want)
        assert torch.equal(ops.dequant_matmul_residual(a.bfloat16(), w, sw, res), (want.float() + res.float()).bfloat16())


@pytest.mark.parametrize("dt", ["bf16", "f16"])
@pytest.mark.parametrize("m,n,k", [(33, 130, 48), (333, 2560, 2048), (777, 3001, 2064), (2047, 1000, 512)])
def test_prompt_product_rounds_like_float64(dt, m, n, k):
    """Two limbs hold 15 bits of the row maximum, so the error of a sum of k random terms stays near sqrt(k) 2^-16 max|a| |w|, far below the
    rounding of the result; a non-finite row spoils itself alone."""
    g = gen(m + 1)
    w, s, act = int8(g, n, k), scales(g, n, DT[dt]), randn(g, m, k).to(DT[dt])
    act[m // 2] = 0
    act[m - 1, 3] = float("nan")
    got, want = ops.dequant_matmul(act, w, s), act.double() @ w.double().t() * s.double()
    assert torch.isnan(got[m - 1]).all()
    ulp = 2.0 ** (-7 if dt == "bf16" else -10)
    assert (got[:-1].double() - want[:-1]).abs().max() <= ulp * want[:-1].abs().max()


# ---- lean products: rows of weights that begin on 32 bytes are read in pieces of 32, others in pieces of 16; the same sums, so the same bits ----
@pytest.mark.parametrize("m", [1, 2, 5])
@pytest.mark.parametrize("n,k", [(300, 1024), (300, 1056), (1121, 2048), (37, 2080), (700, 4096), (145, 4128), (260, 5632)])
def test_lean_products_of_aligned_and_unaligned_rows(m, n, k):
    g = gen(n + k)
    w, s, act = int8(g, n, k), scales(g, n, torch.bfloat16), randn(g, m, k).bfloat16()
    moved = torch.empty(n * k + 16, dtype=torch.int8, device="cuda")[16:].view(n, k)
    moved.copy_(w)
    assert w.data_ptr() % 32 == 0 and moved.data_ptr() % 32 == 16
    got, want = ops.dequant_matmul(act, w, s), act.double() @ w.double().t() * s.double()
    assert torch.equal(got, ops.dequant_matmul(act, moved, s))
    assert (got.double() - want).abs().max() <= 2.0 ** -7 * want.abs().max()


# ---- products of many rows over unquantised weights: pairs of CTAs own 256 weight rows (gating: 128 outputs) and up to 256 activation rows ----
@pytest.mark.parametrize("dt", ["bf16", "f16"])
@pytest.mark.parametrize("m,n,k", [(33, 1, 8), (97, 64, 72), (128, 65, 448), (257, 129, 392), (300, 257, 64), (513, 200, 1032), (2500, 640, 136)])
def test_dense_products_of_cta_pairs(dt, m, n, k):
    g, word = gen(m + n), torch.zeros(1, dtype=torch.int32, device="cuda")
    act, w = randn(g, m, k).to(DT[dt]), (randn(g, 2 * n, k) * k ** -0.5).to(DT[dt])
    act[m - 1] = float("nan")  # stays in its own row
    full = act.double() @ w.double().t()
    # sums of size one: f32 accumulation (k 2^-24) is nothing beside the rounding of the result
    eps = 2.0 ** (-8 if dt == "bf16" else -11)

    def close(got, want, nan=True):
        assert word.item() == 0 and (not nan or torch.isnan(got[m - 1]).all())
        assert (got[:-1].double() - want[:-1]).abs().max() <= (eps + 1e-5) * want[:-1].abs().max()

    close(ops.dense_matmul(act, w, status=word), full)
    close(ops.dense_matmul(act, w, out_dtype=torch.float32, status=word), full)
    gate, up = full[:, :n], full[:, n:]
    close(ops.dense_matmul(act, w, glu=True, status=word), torch.nn.functional.silu(gate) * up)
    got, extra = ops.dense_matmul_ex(act, w, act_fn=ffi.ACT_SQUARE_RELU, f32_columns=n, status=word)
    close(got, torch.relu(gate).square(), nan=False)  # the larger of NaN and 0 is 0 here
    assert torch.isnan(extra[m - 1]).all() and (extra[:-1].double() - up[:-1]).abs().max() <= 1e-5 * up[:-1].abs().max()


@pytest.mark.parametrize("dt", ["bf16", "f16"])
@pytest.mark.parametrize("rows,inner", [(3, 8), (5, 2056), (2, 8192), (2, 8200), (300, 4096)])
def test_dynamic_quantisation_of_rows(dt, rows, inner):
    x = randn(gen(inner), rows, inner).to(DT[dt]) * 3
    want, want_s, _ = R.dynamic_quantize_linear(x.float().cpu().numpy(), True, True, dt)
    y, s, zp = ops.dynamic_quantize_linear(x)
    assert np.array_equal(y.cpu().numpy(), want) and np.array_equal(s.float().cpu().numpy(), want_s) and not zp.any()


# ---- decode attention: wide CTAs up to 74 (sequence, kv head) pairs, four warps above; rounds of 64 to 256 rows, splits ----
@pytest.mark.parametrize("b,hkv,d", [(1, 1, 64), (37, 2, 64), (38, 2, 64), (9, 8, 128), (10, 8, 128)])
@pytest.mark.parametrize("active", [1, 16, 255, 257, 1025, 2300])
def test_decode_attention_rows(b, hkv, d, active):
    g, G = gen(active), 3
    q, k, v = (randn(g, b, h, n, d).bfloat16() for h, n in ((G * hkv, 1), (hkv, 2304), (hkv, 2304)))
    out = ops.window_attention(q, k, v, d ** -0.5, active, 0, 0.0).view_as(q)
    ops.attention_check()
    kk, vv = (t[:, :, :active].double().repeat_interleave(G, 1) for t in (k, v))
    want = torch.softmax((q.double() @ kk.transpose(2, 3)) * d ** -0.5, -1) @ vv
    # the weights are split into two 16-bit parts, so the rounding of the result to bf16 (2^-9) is what remains
    assert (out.double() - want).abs().max() <= 2.0 ** -8 * want.abs().max()


# ---- norms: few rows, many rows, widths around the number of groups per thread ----
@pytest.mark.parametrize("rows", [1, 148, 149])
@pytest.mark.parametrize("W", [4, 1024, 1028, 2052, 4096, 4100, 8192, 8196])
def test_norms_of_few_and_many_rows(rows, W):
    g = gen(W)
    x, w, b = randn(g, rows, W) * 3 + 40.0, randn(g, W), randn(g, W)  # a mean that is large against the deviations
    xd = x.double()
    ln = (xd - xd.mean(1, keepdim=True)) / torch.sqrt(xd.var(1, unbiased=False, keepdim=True) + 1e-5) * w + b
    out = ops.layer_norm(x, w, b, 1e-5, torch.float32)
    assert (out.double() - ln).abs().max() <= 3e-5 * ln.abs().max()  # 40 / 3 * 2^-24 of the mean, times the largest weight
    sub, y = randn(g, rows, W).bfloat16(), x.clone()
    out = ops.residual_rms_norm(y, sub, w, 1e-5)
    s = xd + sub.double()
    rms = s / torch.sqrt((s * s).mean(1, keepdim=True) + 1e-5) * w
    assert (y.double() - s).abs().max() <= 1e-6 * s.abs().max()
    assert (out.double() - rms).abs().max() <= 2.0 ** -8 * rms.abs().max()


# ---- expert choice: logits per lane 2, 8, 32; one CTA up to 64 tokens ----
@pytest.mark.parametrize("M", [1, 64, 65])
@pytest.mark.parametrize("E,top,groups,keep", [(64, 8, 8, 4), (65, 3, 5, 2), (256, 32, 64, 40), (264, 4, 33, 3), (1024, 8, 64, 5)])
def test_expert_choice(M, E, top, groups, keep):
    z = randn(gen(E + M), M, E)
    z[0, :4] = z[0].max() + 1.0  # equal scores go to the lower expert
    z[0, E // 2] = -0.0
    r = ops.MoeRouting(z, top, groups, keep)
    rows, chosen, weights = r.rows().cpu().numpy().reshape(-1), r.chosen.cpu().numpy(), r.weights.double().cpu().numpy()
    for t in range(M):
        e, w = V.route(z[t].double().cpu().numpy(), top, groups, keep)
        assert chosen[t].tolist() == list(e) and np.abs(weights[t] - w).max() <= 3e-6 * w.max()
    order = np.empty(M * top, int)
    order[rows] = chosen.reshape(-1)  # a permutation, ordered by expert
    assert sorted(rows.tolist()) == list(range(M * top)) and (np.diff(order) >= 0).all()


# ---- products over unquantised weights: sixteen warps up to 148 CTAs, blocks of row tiles ----
@pytest.mark.parametrize("M,N,K", [(1, 2368, 264), (8, 2384, 264), (5, 40, 4104), (3, 2050, 72), (3300, 300, 8192)])
def test_dense_products(M, N, K):
    g = gen(N)
    act, w, status = randn(g, M, K).bfloat16(), randn(g, N, K).bfloat16(), torch.zeros(1, dtype=torch.int32, device="cuda")
    want = act.double() @ w.double().t()
    assert (ops.dense_matmul(act, w, status=status).double() - want).abs().max() <= 2.0 ** -8 * want.abs().max()


# ---- decode attention that rotates and appends the new row itself: wide CTAs, several splits, the new row around their borders ----
@pytest.mark.parametrize("head_dim,kv_heads,batch", [(64, 1, 1), (64, 2, 3), (128, 1, 1), (128, 2, 2)])
def test_fused_append_over_a_long_cache(head_dim, kv_heads, batch):
    """Against the rotation and append in front of the attention, over caches whose rows are given.  Few pairs and 4096 rows: eight warps (head_dim
    128) and sixteen (64), clusters of eight splits, rounds of 128 and 256 rows; the contexts put the new row on both sides of warp, round and split borders."""
    from my_nn_engine_b200 import ffi
    from my_nn_engine_b200.decoder import DecoderModel
    from my_nn_engine_b200.quantize import random_llama_state
    cfg = dict(hidden_size=256, num_hidden_layers=1, num_attention_heads=4 * kv_heads, num_key_value_heads=kv_heads, head_dim=head_dim, intermediate_size=256,
               vocab_size=300, rms_norm_eps=1e-5, rope_theta=1e4)
    state, g = random_llama_state(cfg, seed=2), gen(head_dim)
    shape = (batch, kv_heads, 4096, head_dim)
    k, v = randn(g, *shape).bfloat16(), randn(g, *shape).bfloat16()
    edges = [0, 15, 16, 63, 64, 65, 127, 128, 255, 256, 257, 511, 512, 1023, 1024, 1025, 1151, 1152, 2047, 2048, 2049, 4080, 4094]
    runs = []
    try:
        for fuse in (0, 1):
            ffi.set_option(ffi.OPT_FUSE_ROPE, fuse)
            model = DecoderModel(cfg, state, dtype="bf16", max_seq_len=4096, batch=batch)
            rows = []
            for past in edges:
                model.k_cache[0].copy_(k), model.v_cache[0].copy_(v)
                torch.cuda.synchronize()
                rows.append(model.step(np.arange(batch) + past % 200, past).float().clone())
                rows.append((model.k_cache[0].clone(), model.v_cache[0].clone()))
            runs.append(rows)
            model.close()
    finally:
        ffi.set_option(ffi.OPT_FUSE_ROPE, 1)
    for i, past in enumerate(edges):
        # one layer: the appended rows are the same bits; the softmax sums in another order, and what a rounding of the attention to bf16 does to
        # the logits stays within a few of theirs
        (a, b), (ca, cb) = (r[2 * i] for r in runs), (r[2 * i + 1] for r in runs)
        assert torch.equal(ca[0], cb[0]) and torch.equal(ca[1], cb[1]), past
        assert not torch.equal(ca[0][:, :, past], k[:, :, past]) and torch.equal(ca[0][:, :, past + 1:], k[:, :, past + 1:])
        assert (a - b).abs().max() <= 8 * 2.0 ** -7 * a.abs().max(), past


# ---- streaming steps: rotation and append inside the attention kernel, one CTA or a cluster per kv head, against the kernels of their own and the oracle ----
@pytest.mark.parametrize("dt", ["bf16", "f16"])
@pytest.mark.parametrize("d,batch,window", [(64, 1, 15), (64, 3, 509), (64, 2, 1100), (128, 1, 300), (128, 2, 1300), (64, 30, 90)])
def test_streaming_step_with_the_append_inside(dt, d, batch, window):
    """Rows that the step overwrites, and those that are not live yet, hold NaN and infinities."""
    from my_nn_engine_b200.decoder import DecoderModel
    from my_nn_engine_b200.quantize import random_llama_state
    cfg = dict(hidden_size=256, num_hidden_layers=1, num_attention_heads=6, num_key_value_heads=2 if batch < 30 else 3, head_dim=d, intermediate_size=512, vocab_size=300,
               rms_norm_eps=1e-5, rope_theta=1e4)
    sink, tokens = 4, np.arange(batch) * 37 % 300
    rows, state, model = -(-(sink + window) // 8) * 8, random_llama_state(cfg, seed=7), {}
    try:
        for fused in (1, 0):
            ffi.set_option(ffi.OPT_FUSE_ROPE, fused)  # read when a step is captured
            model[fused] = DecoderModel(cfg, state, dtype=dt, max_seq_len=rows, batch=batch, streaming=(sink, window))
            model[fused].stream(tokens, 0)
    finally:
        ffi.set_option(ffi.OPT_FUSE_ROPE, 1)
    want_step, _ = oracle_steps(cfg, state, dt, batch, rows, streaming=(sink, window))
    g = gen(window)
    for pos in (0, 1, 3, 17, sink + window - 1, sink + window, 3 * window + 5):
        past = [randn(g, *model[1].k_cache[0].shape).to(DT[dt]) for _ in range(2)]
        slot = pos if pos < sink else sink + (pos - sink) % window
        for t in past:
            t[:, :, pos + 1:] = float("nan")
            t[:, :, slot, ::2], t[:, :, slot, 1::2] = float("nan"), float("inf")
        for m in model.values():
            m.k_cache[0].copy_(past[0])
            m.v_cache[0].copy_(past[1])
        torch.cuda.synchronize()
        got, apart = (model[f].stream(tokens, pos).clone().double() for f in (1, 0))
        torch.cuda.synchronize()
        for a, b in zip(*((m.k_cache[0], m.v_cache[0]) for m in model.values())):
            assert torch.equal(a.view(torch.int16), b.view(torch.int16)) and torch.isfinite(a[:, :, slot]).all()
        want = want_step(pos, tokens, dict(k_cache=past[0], v_cache=past[1]))
        # the sums of the attention in another order: a rounding of its output here and there, carried through the rest of the layer
        assert (got - apart).abs().max() <= LAYER[dt] * apart.abs().max(), pos
        assert (got - want).abs().max() <= LAYER[dt] * want.abs().max(), pos
    for m in model.values():
        m.close()


# ---- int8 cache, the same: rounds of 128 rows, one CTA, clusters of whole rounds, more pairs than SMs; the new row anywhere in its tile, also a short one ----
@pytest.mark.parametrize("dt", ["bf16", "f16"])
@pytest.mark.parametrize("batch,hkv,rows", [(1, 1, 128), (2, 1, 40), (3, 2, 136), (1, 2, 2048), (5, 8, 768), (2, 3, 3008), (32, 5, 256)])
def test_int8_step_with_the_append_inside(dt, batch, hkv, rows):
    """The same splits, tiles and sums as with a kernel in front that rotates and quantizes, so the same bits."""
    from my_nn_engine_b200.decoder import DecoderModel
    from my_nn_engine_b200.quantize import random_llama_state
    cfg = dict(hidden_size=256, num_hidden_layers=1, num_attention_heads=2 * hkv, num_key_value_heads=hkv, head_dim=128, intermediate_size=512, vocab_size=300,
               rms_norm_eps=1e-5, rope_theta=1e4)
    tokens, model, g, state = np.arange(batch) * 37 % 300, {}, gen(rows + batch), random_llama_state(cfg, seed=9)
    names = ("k_cache", "v_cache", "k_scale", "v_scale")
    try:
        for fused in (1, 0):
            ffi.set_option(ffi.OPT_FUSE_ROPE, fused)  # read when a step is captured
            model[fused] = DecoderModel(cfg, state, dtype=dt, max_seq_len=rows, batch=batch, kv_int8=True)
            model[fused].step(tokens, 0)
    finally:
        ffi.set_option(ffi.OPT_FUSE_ROPE, 1)
    want_step, _ = oracle_steps(cfg, state, dt, batch, rows, kv_int8=True)
    for pos in sorted({0, 1, 31, 32, 100, 127, rows // 2 + 3, rows - 9, rows - 1}):
        if pos >= rows:
            continue
        past = [int8(g, *model[1].k_cache[0].shape) for _ in range(2)] + [scales(g, model[1].k_scale[0].numel(), DT[dt]).view_as(model[1].k_scale[0]) for _ in range(2)]
        for m in model.values():
            for name, t in zip(names, past):
                getattr(m, name)[0].copy_(t)
        torch.cuda.synchronize()
        got, apart = (model[f].step(tokens, pos).clone().double() for f in (1, 0))
        torch.cuda.synchronize()
        for name in names:
            assert torch.equal(getattr(model[1], name)[0], getattr(model[0], name)[0])
        assert torch.equal(got, apart), pos
        want = want_step(pos, tokens, dict(zip(names, past)))
        assert (got - want).abs().max() <= LAYER[dt] * want.abs().max(), pos
    for m in model.values():
        m.close()


# ---- more sequences than the lean products take: the attention leaves its rows as limbs, behind the merge of a cluster too ----
@pytest.mark.parametrize("dt", ["bf16", "f16"])
@pytest.mark.parametrize("d,batch,hkv,rows", [(128, 6, 1, 1024), (64, 6, 1, 2048), (128, 9, 2, 1536), (64, 20, 1, 1536)])
def test_clusters_leave_limbs_like_the_oracle(dt, d, batch, hkv, rows):
    """Both sides of the two rounds (256 rows of eight warps, 512 of sixteen) that a cluster leaves to its first CTA."""
    from my_nn_engine_b200.decoder import DecoderModel
    from my_nn_engine_b200.quantize import random_llama_state
    cfg = dict(hidden_size=256, num_hidden_layers=1, num_attention_heads=4 * hkv, num_key_value_heads=hkv, head_dim=d, intermediate_size=512, vocab_size=300,
               rms_norm_eps=1e-5, rope_theta=1e4)
    state, g, tokens = random_llama_state(cfg, seed=3), gen(rows + d), np.arange(batch) * 37 % 300
    model = DecoderModel(cfg, state, dtype=dt, max_seq_len=rows, batch=batch)
    want_step, _ = oracle_steps(cfg, state, dt, batch, rows)
    for pos in (0, 70, 254, 255, 256, 511, 512, 513, 900, rows - 1):
        past = [randn(g, *model.k_cache[0].shape).to(DT[dt]) for _ in range(2)]
        model.k_cache[0].copy_(past[0])
        model.v_cache[0].copy_(past[1])
        torch.cuda.synchronize()
        got, want = model.step(tokens, pos).clone().double(), want_step(pos, tokens, dict(k_cache=past[0], v_cache=past[1]))
        assert (got - want).abs().max() <= LAYER[dt] * want.abs().max(), pos
    model.close()


# ---- windows over a ring: clusters whose first visible row lies inside a tile, rows on both sides of the two rounds that one CTA takes ----
@pytest.mark.parametrize("dt", ["bf16", "f16"])
@pytest.mark.parametrize("d,window", [(128, 241), (128, 255), (128, 256), (128, 257), (128, 700), (64, 497), (64, 511), (64, 512), (64, 513), (64, 1000)])
def test_windows_that_clusters_share(dt, d, window):
    g, rows, batch, hkv, hq = gen(window), 1024, 2, 2, 6
    q, k, v = (randn(g, batch, h, n, d).to(DT[dt]) for h, n in ((hq, 1), (hkv, rows), (hkv, rows)))
    for active in (window - 3, window + 5, 800, 1000, 1024, 1031, 5003):
        at = torch.arange(max(0, active - window), active) % rows
        kk, vv = (t[:, :, at].double().repeat_interleave(hq // hkv, 1) for t in (k, v))
        for cap in (0.0, 6.0):
            s = q.double() @ kk.transpose(2, 3) * d ** -0.5
            want = ((cap * torch.tanh(s / cap) if cap else s).softmax(-1) @ vv).transpose(1, 2)
            got = ops.window_attention(q, k, v, d ** -0.5, active, window, cap)
            # weights carry 16 bits, the soft cap 2^-10 of itself; what counts is the rounding of the output
            assert (got.double() - want).abs().max() <= {"bf16": 2.0 ** -7, "f16": 2.0 ** -9}[dt] * want.abs().max(), (active, cap)


# ---- products of experts on pairs of CTAs: experts of one tile, of one and a row, and rows of another expert that a tile's copies bring along ----
@pytest.mark.parametrize("dt", ["bf16", "f16"])
@pytest.mark.parametrize("sizes", [(256, 257, 31, 56), (0, 512, 1, 33), (225, 32, 513, 16)])
def test_experts_of_whole_tiles_keep_to_their_rows(dt, sizes):
    n, k, experts = 130, 72, len(sizes)
    g, of = gen(sum(sizes)), torch.repeat_interleave(torch.arange(experts), torch.tensor(sizes))
    of = of[torch.randperm(len(of), generator=torch.Generator().manual_seed(1))].cuda()
    routing = ops.MoeRouting(torch.nn.functional.one_hot(of, experts).float() * 9, 1)
    place = routing.rows().reshape(-1).long()
    act, gu, dn = randn(g, len(of), k).to(DT[dt]), (randn(g, experts, 2 * n, k) * k ** -0.5).to(DT[dt]), (randn(g, experts, k, n) * n ** -0.5).to(DT[dt])
    hidden = randn(g, len(of), n).to(DT[dt])

    def run(a, h):
        out = []
        for args in (dict(act=a, w=gu, gather=True, glu=True), dict(act=h, w=dn, gather=False, out_dtype=torch.float32)):
            out.append(routing.matmul(**args))
            assert int(routing.status.item()) == 0
        return out

    clean = run(act, hidden)
    by_place = torch.empty_like(of)
    by_place[place] = of
    for e in range(experts):
        full = act[of == e].double() @ gu[e].double().t()
        want = torch.nn.functional.silu(full[:, :n]) * full[:, n:]
        eps = 2.0 ** (-8 if dt == "bf16" else -11)
        if len(want):
            assert (clean[0][place[of == e]].double() - want).abs().max() <= (eps + 1e-5) * want.abs().max()
            want = hidden[by_place == e].double() @ dn[e].double().t()
            assert (clean[1][by_place == e].double() - want).abs().max() <= 1e-5 * want.abs().max()
        bad_act, bad_hidden = act.clone(), hidden.clone()
        bad_act[of == e], bad_hidden[by_place == e] = float("nan"), float("nan")
        for got, was in zip(run(bad_act, bad_hidden), clean):
            assert torch.isnan(got[by_place == e]).all() and torch.equal(got[by_place != e], was[by_place != e])


# ---- decode attention whose splits meet: scores that are NaN in all rows of a warp or of a split are not lost, and stay with their sequence ----
@pytest.mark.parametrize("form", ["int8", "plain", "window"])
@pytest.mark.parametrize("d,batch,rows", [(64, 2, 64), (128, 3, 512), (64, 2, 2048), (128, 2, 2048), (64, 2, 3072), (128, 20, 1024), (128, 2, 40960)])
def test_nan_rows_reach_the_output_through_every_merge(form, d, batch, rows):
    """One CTA; clusters of two to eight splits; through L2 (40960 rows, 16 splits).  Only a range of whole splits shows a loss."""
    hq, g, scale, dt = 4, gen(rows + d), d ** -0.5, torch.bfloat16
    q, k, v = randn(g, batch, hq, 1, d).to(dt), randn(g, batch, 2, rows, d).to(dt), randn(g, batch, 2, rows, d).to(dt)
    if form == "int8":
        k, v, ks, vs = int8(g, *k.shape), int8(g, *k.shape), *(scales(g, batch * 2 * rows, dt).view(batch, 2, rows) for _ in range(2))

    def run(where):
        if form == "int8":
            bad = ks.clone()
            bad[1, 0, where] = float("nan")
            return ops.attention_q8(q, k, v, bad, vs, scale)
        bad = k.clone()
        bad[1, 0, where] = float("nan")
        return ops.attention(q, bad, v, scale) if form == "plain" else ops.window_attention(q, bad, v, scale, rows).transpose(1, 2)

    clean = run(slice(0, 0))
    assert torch.isfinite(clean).all()
    for where in (slice(0, 16), slice(0, rows // 8 * 3), slice(0, rows // 2), slice(rows // 4, rows // 2), slice(rows // 2, rows), slice(rows - 1, rows)):
        got, want = run(where), clean.clone()
        want[1, :hq // 2] = float("nan")
        assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.nan_to_num(), want.nan_to_num()), where
