"""Prompts taken a layer at a time with the recurrence in token order (fp32 weights, short prompts, other head shapes) against
the same prompt token by token, and against the oracle."""
import numpy as np
import pytest

import lumi_b200
from lumi_b200 import synth
from oracle import cpu_oracle

pytestmark = pytest.mark.gpu


def rel(a, b):
    return float(np.abs(a - b).max() / np.abs(b).max())


def pair(cfg, dtype, batch, seed=3):
    tens = list(synth.iter_tensors(cfg, seed=seed, weights_dtype=dtype, perturb_ones=0.1))
    model = lumi_b200.NmModel.from_tensors(cfg, tens)
    rows, steps = model.init_states(batch, 256), model.init_states(batch, 256)
    steps.set_option("chunked_prefill", 0)
    return tens, model, rows, steps


def same_state(rows, steps, b, layer, tol):
    for x, y, what in zip(rows.read_state(b, layer), steps.read_state(b, layer), ("h", "x_prev", "b_prev", "angle")):
        if what == "angle":
            x = y + np.mod(x - y + np.pi, 2 * np.pi) - np.pi
        assert np.abs(x - y).max() <= tol * max(1.0, np.abs(y).max()), (b, layer, what)


# Sums of at most 512 products in two orders: 512 * 2^-24 = 3e-5 of the sum of magnitudes at the very worst, a tenth of it in practice;
# bf16 models of nine sequences and more round activations to two bf16 halves (2^-17 per factor) on both sides, after sums in two orders.
TOL = {"f32": 3e-5, "bf16": 2e-4}


# Without this the comparisons below could hold steps against steps.  A step is at least four launches per layer and token, a pass five per layer.
@pytest.mark.parametrize("dtype,batch,T,kw,taken", [
    ("f32", 1, 4, {}, False), ("f32", 1, 8, {}, True), ("f32", 3, 4, {}, True), ("f32", 13, 5, {}, True), ("f32", 4, 40, dict(n_heads=16, d_state=16), False),
    ("f32", 4, 40, dict(n_heads=16, d_state=32), True), ("f32", 4, 40, dict(n_heads=4, d_state=128), True), ("f32", 4, 40, dict(attention_interval=2), False),
    ("bf16", 1, 4, {}, False), ("bf16", 1, 6, {}, True), ("bf16", 3, 4, {}, True), ("bf16", 13, 4, {}, True), ("bf16", 13, 3, {}, False),
    ("bf16", 2, 5, dict(attention_interval=2, attn_rope_base=10000.0), True)])
def test_which_prompts_go_a_layer_at_a_time(dtype, batch, T, kw, taken):
    cfg = synth.tiny_config(**{**dict(n_layers=3), **kw})
    _, _, rows, steps = pair(cfg, dtype, batch)
    prompts = synth.random_prompts(batch, T, cfg.vocab_size, seed=T)
    launches = [s.generate(prompts, 1, ignore_eos=True)[3].kernel_launches for s in (rows, steps)]
    assert (launches[0] < launches[1]) == taken, launches
    assert taken or launches[0] == launches[1]


# tokens around the sixteen that are taken at a time, rows around the tiles of 32 and 64, K split and not
@pytest.mark.parametrize("dtype", ["f32", "bf16"])
@pytest.mark.parametrize("batch,T", [(1, 4), (1, 15), (1, 16), (1, 17), (1, 33), (2, 32), (3, 22), (5, 65), (13, 5), (20, 33)])
def test_rows_equal_steps(dtype, batch, T):
    cfg = synth.tiny_config(n_layers=3)
    tens, _, rows, steps = pair(cfg, dtype, batch)
    prompts = synth.random_prompts(batch, T, cfg.vocab_size, seed=T)
    assert rel(rows.prefill(prompts), steps.prefill(prompts)) < TOL[dtype]
    for layer in range(cfg.n_layers):
        same_state(rows, steps, batch - 1, layer, 10 * TOL[dtype])
    # a second prompt behind the first starts from the handed-over state, and the oracle agrees with both
    more = synth.random_prompts(batch, 5, cfg.vocab_size, seed=T + 1)
    a, b = rows.prefill(more), steps.prefill(more)
    assert rel(a, b) < TOL[dtype]
    st = cpu_oracle.OracleModel(cfg, tens).init_states()
    for tok in np.concatenate([prompts[-1], more[-1]]):
        ref = st.forward_step(int(tok))
    assert rel(a[-1], ref) < TOL[dtype]


@pytest.mark.parametrize("heads,d_state", [(8, 32), (8, 64), (8, 128), (16, 32), (16, 64), (16, 128), (4, 16), (4, 32), (4, 64), (4, 128), (16, 16)])
def test_rows_of_every_head_shape(heads, d_state):
    """Head widths 64, 32 and 16 (16 x 16 is the one that stays with the steps)."""
    cfg = synth.tiny_config(n_layers=2, n_heads=heads, d_state=d_state)
    _, _, rows, steps = pair(cfg, "f32", 3)
    prompts = synth.random_prompts(3, 37, cfg.vocab_size, seed=heads + d_state)
    assert rel(rows.prefill(prompts), steps.prefill(prompts)) < TOL["f32"]
    for layer in range(2):
        same_state(rows, steps, 1, layer, 10 * TOL["f32"])


@pytest.mark.parametrize("dtype", ["f32", "bf16"])
def test_rows_of_different_lengths_and_scores(dtype):
    cfg = synth.tiny_config(n_layers=3)
    _, _, rows, steps = pair(cfg, dtype, 4)
    prompts = synth.random_prompts(4, 40, cfg.vocab_size, seed=8)
    lengths = np.array([40, 1, 16, 33], dtype=np.int32)
    assert rel(rows.prefill_ragged(prompts, lengths), steps.prefill_ragged(prompts, lengths)) < TOL[dtype]
    for b in range(4):
        same_state(rows, steps, b, 1, 10 * TOL[dtype])
    rows.reset(), steps.reset()
    a, b = rows.score(prompts), steps.score(prompts)
    assert np.abs(a - b).max() < 10 * TOL[dtype] * np.abs(b).max()
    assert np.array_equal(rows.forward_step(prompts[:, 0])[1], steps.forward_step(prompts[:, 0])[1])


@pytest.mark.parametrize("T", [5, 30])
def test_short_prompts_with_attention_layers(T):
    cfg = synth.tiny_config(attention_interval=2, attn_rope_base=10000.0)
    _, _, rows, steps = pair(cfg, "bf16", 2)
    prompts = synth.random_prompts(2, T, cfg.vocab_size, seed=T)
    assert rel(rows.prefill(prompts), steps.prefill(prompts)) < 2e-3          # the two sides round their keys and values to bf16 on their own
    assert rel(rows.forward_step(prompts[:, 0])[0], steps.forward_step(prompts[:, 0])[0]) < 2e-3


# up to eight bf16 sequences take fp32 activations token by token, and have to as prompts: two bf16 halves (2^-17 of each factor, 8e-6) would show
# against sums in another order (at most 512 products, 512 * 2^-24 = 3e-5 at the very worst, a tenth of it in practice)
@pytest.mark.parametrize("batch,T", [(1, 6), (1, 90), (3, 33), (8, 20)])
@pytest.mark.parametrize("split", [1, 0])
def test_few_bf16_sequences_keep_fp32_activations(batch, T, split):
    cfg = synth.tiny_config(n_layers=3)
    _, _, rows, steps = pair(cfg, "bf16", batch)
    for s in (rows, steps):
        s.set_option("split_activations", split)
    prompts = synth.random_prompts(batch, T, cfg.vocab_size, seed=T)
    a, b = rows.prefill(prompts), steps.prefill(prompts)
    assert rel(a, b) < 3e-6
    rows.reset(), steps.reset()
    a, b = rows.score(prompts), steps.score(prompts)
    assert np.abs(a - b).max() < 3e-6 * np.abs(b).max()


# a slice's rows count from the prompt's first token, the cache from the sequence's: first prompts of different lengths, so that the two differ by
# another amount in every sequence; lengths of one token, of the longest, around a slice of 64; tensor-core and CUDA-core attention
@pytest.mark.parametrize("kv_heads,heads", [(4, 16), (8, 32)])
@pytest.mark.parametrize("T", [30, 140])
def test_ragged_prompts_behind_earlier_tokens(T, kv_heads, heads):
    cfg = synth.base_config(n_layers=3, vocab_size=700, attention_layers=[1], attn_mlp_dim=256, attn_rope_base=10000.0, attn_n_heads=heads, attn_kv_heads=kv_heads)
    _, _, rows, steps = pair(cfg, "bf16", 4)
    rows.set_option("prefill_rows", 256)
    first = synth.random_prompts(4, 40, cfg.vocab_size, seed=1)
    second = synth.random_prompts(4, T, cfg.vocab_size, seed=2)
    lengths = np.array([T, 1, min(T, 64), min(T, 65)], dtype=np.int32)
    for prompts, lens in ((first, np.array([40, 7, 33, 40], dtype=np.int32)), (second, lengths)):
        a, b = rows.prefill_ragged(prompts, lens), steps.prefill_ragged(prompts, lens)
        assert rel(a, b) < 2e-3                            # keys and values are rounded to bf16 on each side
    for i in range(3):
        a, b = (s.forward_step(second[:, i], step=i)[0] for s in (rows, steps))
        for j in range(4):
            assert rel(a[j], b[j]) < 2e-3, (i, j)


# 16 x 160 rows of 41 KB: in one pass with room for it, in smaller passes, and token by token without room for the smallest (512 rows, 21 MB)
@pytest.mark.parametrize("op", ["prefill", "score"])
@pytest.mark.parametrize("left_mb,fits", [(None, True), (64, True), (12, False)])
def test_prompts_where_there_is_little_memory(op, left_mb, fits):
    import torch
    cfg = synth.base_config(n_layers=2, vocab_size=500)
    tens = list(synth.iter_tensors(cfg, seed=3, weights_dtype="f32", perturb_ones=0.1))
    model = lumi_b200.NmModel.from_tensors(cfg, tens)
    warm, rows, steps = (model.init_states(16, 256) for _ in range(3))
    steps.set_option("chunked_prefill", 0)
    rows.set_option("graph", 0)                              # captured graphs take memory of their own
    prompts = synth.random_prompts(16, 160, cfg.vocab_size, seed=5)
    want = getattr(steps, op)(prompts)
    getattr(warm, op)(prompts)                               # every kernel is loaded
    warm.close()
    hold = []
    try:
        if left_mb is not None:                              # blocks of 32 MB and more come straight from the device
            spare = torch.cuda.mem_get_info()[0] - (left_mb << 20)
            hold = [torch.empty(1 << 30, dtype=torch.uint8, device="cuda") for _ in range((spare >> 30) - 1)]
            spare = torch.cuda.mem_get_info()[0] - (left_mb << 20)
            hold.append(torch.empty(spare >> 21 << 21, dtype=torch.uint8, device="cuda"))
        got = getattr(rows, op)(prompts)
    finally:
        del hold
        torch.cuda.empty_cache()
    if fits:
        assert rel(got, want) < TOL["f32"] * (10 if op == "score" else 1)
    else:
        assert np.array_equal(got, want)
    assert rel(rows.forward_step(prompts[:, 0])[0], steps.forward_step(prompts[:, 0])[0]) < TOL["f32"]
