"""GPU: the gate of an attention block's MLP takes two quads per thread, in prompts and in steps, at widths that fill its blocks or not;
results of the state step where it asks for states one block per SM ahead, over heads that do not fill their last block (the requests
themselves change no result; the gate's own values: test_gpu_gate_values.py).

Bound: the benchmark definition's 2e-2 of the largest logit for bf16 weights (the cache of keys and values is bf16)."""
import numpy as np
import pytest

import lumi_b200
from lumi_b200 import synth
from oracle import cpu_oracle
from tests.helpers import rel_err

pytestmark = pytest.mark.gpu

TOL_BF16 = 2e-2


def _check(cfg, batch, T, n_new):
    tens = list(synth.iter_tensors(cfg, seed=8, weights_dtype="bf16", perturb_ones=0.1))
    prompts = synth.random_prompts(batch, T, cfg.vocab_size, seed=3)
    model = lumi_b200.NmModel.from_tensors(cfg, tens)
    toks, _, dump, _ = model.init_states(batch, T + n_new).generate(prompts, n_new, ignore_eos=True, dump_logits=True)
    om = cpu_oracle.OracleModel(cfg, tens)
    for b in (0, batch // 2, batch - 1):
        ref_toks, ref_logits = om.init_states().generate(prompts[b], n_new, ignore_eos=True, dump_logits=True)
        n_same = n_new if np.array_equal(toks[b], ref_toks) else int(np.argmax(toks[b] != ref_toks)) + 1
        assert max(rel_err(dump[i, b], ref_logits[i]) for i in range(n_same)) < TOL_BF16


@pytest.mark.parametrize("width", [8, 1032, 2056, 2816])      # 2, 258, 514 and 704 quads: one block, one, two, two
def test_gate_widths(width):
    _check(synth.tiny_config(n_layers=2, attention_layers=[1], attn_mlp_dim=width), 12, 40, 3)


@pytest.mark.parametrize("batch", [12, 60])                       # 36 blocks: none is a block per SM ahead; 180: some are
def test_states_asked_for_ahead(batch):
    _check(synth.tiny_config(n_layers=2, d_model=320, n_heads=20, d_state=64), batch, 3, 4)
