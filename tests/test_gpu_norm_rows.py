"""GPU: the norm in front of a prompt's products has two kernels, one for few and one for many rows; they give the same bits."""
import numpy as np
import pytest

import lumi_b200
from lumi_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("d_model,n_heads", [(128, 8), (320, 20)])
def test_many_rows_have_the_bits_of_few(d_model, n_heads):
    cfg = synth.tiny_config(n_layers=2, d_model=d_model, n_heads=n_heads, d_state=64)
    model = lumi_b200.NmModel.from_tensors(cfg, list(synth.iter_tensors(cfg, seed=3, weights_dtype="bf16")))
    batch, T = 18, 131                                        # 2358 rows, and 1179 in each half
    prompts = synth.random_prompts(batch, T, cfg.vocab_size, seed=4)
    whole = model.init_states(batch, T + 2).prefill(prompts)
    for half in (slice(0, 9), slice(9, 18)):
        sess = model.init_states(9, T + 2)
        assert np.array_equal(sess.prefill(prompts[half]), whole[half])
