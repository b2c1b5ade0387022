"""Operators queued one behind the other without a host synchronisation: what one writes is what the next reads, whichever operand it is."""
import pytest
import torch

pytestmark = pytest.mark.gpu

from my_nn_engine_b200 import ffi, ops  # noqa: E402

DT = {"bf16": torch.bfloat16, "f16": torch.float16}


def randn(seed, *shape):
    return torch.randn(*shape, generator=torch.Generator(device="cuda").manual_seed(seed), device="cuda")


def quantise_into(q, s, zp, w):
    ffi.check(ffi.lib().mynn_b200_dynamic_quantize_linear(ops._stream(), q.data_ptr(), s.data_ptr(), zp.data_ptr(), w.data_ptr(), *w.shape, 1, 1, ops._dt(w)))


# rows of W: fewer than SMs, a ragged last wave, many waves; k of every form of the products and, at 8208, past the quantiser for short rows
@pytest.mark.parametrize("dt", ["bf16", "f16"])
@pytest.mark.parametrize("n,k", [(64, 2048), (1000, 512), (1000, 8192), (1000, 8208), (5632, 2048), (20000, 4096)])
def test_weights_quantised_right_in_front_of_the_product(dt, n, k):
    """DynamicQuantizeLinear makes int8 rows and one scale per row, which is what DequantMatMul takes as weights.  One launch after the other,
    with work in front so that the host is ahead, and replayed from a graph, the product has the bits of the synchronised sequence."""
    w, other = randn(n, n, k).to(DT[dt]), randn(n + 1, n, k).to(DT[dt])
    acts = [randn(m, m, k).to(DT[dt]) for m in (1, 2, 3, 5, 8, 32, 40)]
    res = [randn(n + a.shape[0], a.shape[0], n).to(DT[dt]) for a in acts]
    q, s, zp = ops.dynamic_quantize_linear(w)
    torch.cuda.synchronize()
    want = [(ops.dequant_matmul(a, q, s), ops.dequant_matmul_residual(a, q, s, r)) for a, r in zip(acts, res)]
    torch.cuda.synchronize()
    busy = randn(0, 4096, 4096)

    def once():
        got = []
        for a, r in zip(acts, res):
            quantise_into(q, s, zp, other)  # stale weights and scales for the next two
            quantise_into(q, s, zp, w)
            x = ops.dequant_matmul(a, q, s)
            quantise_into(q, s, zp, other)
            quantise_into(q, s, zp, w)
            got.append((x, ops.dequant_matmul_residual(a, q, s, r)))
        return got

    for _ in range(3):
        busy @ busy
        for (x, y), (x0, y0) in zip(once(), want):
            assert torch.equal(x, x0) and torch.equal(y, y0)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = once()
    for _ in range(3):
        graph.replay()
    torch.cuda.synchronize()
    for (x, y), (x0, y0) in zip(got, want):
        assert torch.equal(x, x0) and torch.equal(y, y0)


@pytest.mark.parametrize("m", [1, 3, 8, 32])
def test_second_matrix_quantised_right_in_front_of_its_product(m):
    """dequant_matmul_same_act: the activations' limbs come from the call before, the weights from the kernel right in front."""
    n, k = 1500, 2048
    a, w1, w2 = randn(1, m, k).bfloat16(), randn(2, n, k).bfloat16(), randn(3, n, k).bfloat16()
    q1, s1, _ = ops.dynamic_quantize_linear(w1)
    q2, s2, zp = ops.dynamic_quantize_linear(w2)
    torch.cuda.synchronize()
    want = ops.dequant_matmul(a, q2, s2)
    torch.cuda.synchronize()
    busy = randn(0, 4096, 4096)
    for _ in range(5):
        busy @ busy
        ops.dequant_matmul(a, q1, s1)
        quantise_into(q2, s2, zp, w1)
        quantise_into(q2, s2, zp, w2)
        assert torch.equal(ops.dequant_matmul_same_act(a, q2, s2), want)


@pytest.mark.parametrize("heads,kv_heads,head_dim", [(4, 2, 64), (4, 1, 128)])
def test_int8_cache_row_rewritten_below_the_last_visible_one(heads, kv_heads, head_dim):
    """A step may write a row in the middle of the rows it attends to (past_len below active_seq_kv - 1).  The row holds something else before
    the first pass and its own bytes before the second, so the two agree only if the attention takes the row that the step wrote."""
    from my_nn_engine_b200.decoder import DecoderModel
    from my_nn_engine_b200.quantize import random_llama_state
    cfg = dict(hidden_size=heads * head_dim, num_hidden_layers=3, num_attention_heads=heads, num_key_value_heads=kv_heads, head_dim=head_dim, intermediate_size=512,
               vocab_size=300, rms_norm_eps=1e-5, rope_theta=1e4)
    model = DecoderModel(cfg, random_llama_state(cfg, seed=1), dtype="bf16", max_seq_len=2048, batch=2, kv_int8=True)
    for i in range(3):
        for cache, scale in ((model.k_cache[i], model.k_scale[i]), (model.v_cache[i], model.v_scale[i])):
            cache.copy_((randn(i, *cache.shape) * 40).clamp(-127, 127).to(torch.int8))
            scale.fill_(0.02)
    for past in (0, 31, 32, 700, 1023, 1030, 1999):
        for i in range(3):
            for cache, scale in ((model.k_cache[i], model.k_scale[i]), (model.v_cache[i], model.v_scale[i])):
                cache[:, :, past] = 127
                scale[:, :, past] = 3.0
        torch.cuda.synchronize()
        first = model.step([5, 7], past, 2000).clone()
        for _ in range(3):
            assert torch.equal(model.step([5, 7], past, 2000), first)
    model.close()


def llama(kv_int8, use_graph):
    from my_nn_engine_b200.decoder import DecoderModel
    from my_nn_engine_b200.quantize import random_llama_state
    cfg = dict(hidden_size=256, num_hidden_layers=4, num_attention_heads=2, num_key_value_heads=1, head_dim=128, intermediate_size=512, vocab_size=300,
               rms_norm_eps=1e-5, rope_theta=1e4)
    state = random_llama_state(cfg, seed=1)
    return 300, lambda: DecoderModel(cfg, state, dtype="bf16", max_seq_len=512, batch=2, kv_int8=kv_int8, use_graph=use_graph)


def blocks(family, name, use_graph):
    from my_nn_engine_b200 import fimadra, vebisun
    from tests import block_models as bm
    from tests import fimadra_models as fm
    lib, models = (fimadra, fm) if family == "fimadra" else (vebisun, bm)
    cfg = getattr(models, name)()
    state = models.weights(cfg, seed=1)
    return cfg["vocab"], lambda: lib.build(cfg, state, dtype="bf16", max_seq_len=512, batch=2, use_graph=use_graph)


@pytest.mark.parametrize("use_graph", [False, True])
@pytest.mark.parametrize("make", [lambda g: llama(False, g), lambda g: llama(True, g), lambda g: blocks("vebisun", "even_group", g), lambda g: blocks("vebisun", "odd_group", g),
                                  lambda g: blocks("fimadra", "chunkwise", g), lambda g: blocks("fimadra", "wide", g)])
def test_queued_steps_equal_synchronised_ones(make, use_graph):
    """What a step reads ahead of its kernels (cached rows, memories, conv history, positions) is what the step before it has left, also when
    the steps are queued one behind the other."""
    vocab, build = make(use_graph)
    steps = 300
    ids = torch.randint(0, vocab, (steps, 2), generator=torch.Generator().manual_seed(3)).cuda()
    outs, stream = [], torch.cuda.Stream()
    for synchronise in (True, False):
        model = build()
        out = torch.empty(steps, 2, vocab, dtype=model._logits_dtype, device="cuda")
        torch.cuda.synchronize()
        for i in range(steps):
            model.step_device(ids[i], i, out[i], stream.cuda_stream)
            if synchronise:
                torch.cuda.synchronize()
        torch.cuda.synchronize()
        outs.append(out)
        model.close()
    assert torch.isfinite(outs[0].float()).all() and torch.equal(outs[0], outs[1])
