"""GPU: which tokens survive top-k and which one is drawn, where values tie and where the row is short."""
import numpy as np
import pytest

import lumi_b200
from lumi_b200 import synth
from oracle import numpy_restatement as nr

pytestmark = pytest.mark.gpu


# groups: how many different embedding rows there are (ids share them in turn, so their logits are equal bit by bit).  One group: more ties
# than the selection lists (1024), which falls back to the histograms; rows shorter and longer than the block; k of 1, of most, of the largest
@pytest.mark.parametrize("V,groups", [(300, 300), (1000, 40), (1025, 1025), (5000, 7), (3000, 1), (32000, 32000), (32000, 3000)])
@pytest.mark.parametrize("k", [1, 50, 256])
def test_tied_and_short_rows(V, groups, k):
    cfg = synth.tiny_config(n_layers=1, vocab_size=V)
    tens = []
    for name, dt, a in synth.iter_tensors(cfg, seed=3):
        if name.endswith("embedding.weight"):
            a = np.ascontiguousarray(a[np.arange(V) % groups]) * np.float32(3.0)
        tens.append((name, dt, a))
    sess = lumi_b200.NmModel.from_tensors(cfg, tens).init_states(2)
    tok = np.array([5, 17], dtype=np.uint32) % V
    for step in range(6):
        sp = lumi_b200.Sampling(0.8, k, 4321, 2, 1)
        logits, nxt = sess.forward_step(tok, sampling=sp, step=step)
        for b in range(2):
            r = nr.sampler_uniform(4321, b, step)
            want = nr.sample_from_logits(logits[b], 0.8, k, r)
            if int(nxt[b]) == want:
                continue
            # expf of the GPU and of numpy differ in the last bit: another pick only where the cumulative sum meets the uniform, and a survivor
            order = np.argsort(-logits[b], kind="stable")[:k]
            assert int(nxt[b]) in order
            kept = np.sort(order)
            p = np.exp((logits[b][kept] * np.float32(1 / 0.8)).astype(np.float64))
            assert np.abs(np.cumsum(p / p.sum()) - float(r)).min() < 1e-5
        tok = nxt
