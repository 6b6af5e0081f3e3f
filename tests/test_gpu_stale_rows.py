"""GPU: prompts of different lengths after a call that left no numbers in every buffer of the session.  Products skip blocks of 32 rows behind a prompt's end, so
what an earlier call left there is still there when the kernels behind them run; nothing of it may reach a result."""
import numpy as np
import pytest

import lumi_b200
from lumi_b200 import synth, zozonex as zz, zutazen as zt

pytestmark = pytest.mark.gpu
BATCH, T = 12, 200                                            # 2400 rows: above 1024 the row blocks are taken


def _model(design):
    if design == "hybrid":
        cfg = synth.tiny_config(n_layers=3, d_model=256, n_heads=16, d_state=64, attention_layers=[1], attn_mlp_dim=512)
        return cfg, list(synth.iter_tensors(cfg, seed=6, weights_dtype="bf16", perturb_ones=0.1))
    if design == "zozonex":
        cfg = zz.config(128, 256, [zz.delta(4, 64, 128), zz.attention(4, 64, 70, kv_heads=2, ff=256), zz.delta(4, 64, 128, ff=256)])
        return cfg, list(zz.iter_tensors(cfg, seed=6))
    # (widths in whole k-blocks of 64: the columns that fill up a block of another width are not written again by every call)
    mlp = zt.dense(256)
    cfg = zt.config(128, 256, [zt.retention(2, 128, 128, mlp=mlp), zt.rglru(128, 2, mlp=zt.moe(8, 2, 64)), zt.latent_attention(4, 64, 32, 64, 128, 70, mlp=mlp),
                               zt.rglru(128, 2, mlp=mlp)])
    return cfg, list(zt.iter_tensors(cfg, seed=6))


@pytest.mark.parametrize("design", ["hybrid", "zozonex", "zutazen"])
def test_nothing_of_an_earlier_call_is_seen(design):
    cfg, tens = _model(design)
    tens = [(n, dt, a.copy()) for n, dt, a in tens]
    (dt, emb), = [(dt, a) for n, dt, a in tens if n.endswith(("embed", "embedding.weight"))]
    emb[0] = 0x7fc0 if dt == synth.BF16 else np.nan           # token 0 has no numbers
    model = lumi_b200.NmModel.from_tensors(cfg, tens)
    g = np.random.default_rng(5)
    prompts = g.integers(1, cfg.vocab_size, (BATCH, T)).astype(np.uint32)
    lens = np.array([T, 1, 31, 32, 33, 64, 65, 90, 5, 150, 2, 17], np.int32)
    results = []
    for used in (False, True):
        sess = model.init_states(BATCH, T + 8)
        if used:
            sess.prefill(np.zeros((BATCH, T), np.uint32), want_logits=False)
            sess.reset()
        logits = sess.prefill_ragged(prompts, lens)
        assert np.isfinite(logits[:, 1:]).all()               # (a tied head has no number for token 0)
        results.append((logits, [sess.save_state(b) for b in range(BATCH)]))
        sess.close()
    assert np.array_equal(results[0][0], results[1][0], equal_nan=True)
    model.close()
