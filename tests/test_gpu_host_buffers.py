"""GPU: logits into a caller's own buffer: ordinary memory (whose pages are touched ahead of the copy from 64 KiB on) at any address, memory that CUDA pinned or was
told of; nothing beside the buffer changes."""
import ctypes as C

import numpy as np
import pytest

import lumi_b200
from lumi_b200 import synth

pytestmark = pytest.mark.gpu
GUARD = 8192


@pytest.fixture(scope="module")
def session():
    cfg = synth.tiny_config(n_layers=1, vocab_size=8200)      # 32800 bytes of logits a sequence
    model = lumi_b200.NmModel.from_tensors(cfg, list(synth.iter_tensors(cfg, seed=2)))
    sess = model.init_states(8, 16)
    yield sess, synth.random_prompts(8, 3, cfg.vocab_size, seed=3)
    sess.close(); model.close()


# one sequence: below the line; two: 64 bytes above it; eight: 64 pages and a rest
@pytest.mark.parametrize("batch", [1, 2, 8])
@pytest.mark.parametrize("kind,shift", [("fresh", 0), ("fresh", 4), ("fresh", 1), ("fresh", 4095), ("pinned", 0), ("pinned", 12), ("registered", 0), ("registered", 4)])
def test_logits_arrive_and_nothing_else_changes(session, batch, kind, shift):
    import torch
    sess, prompts = session
    sess.reset()
    want = sess.prefill(prompts[:batch])
    n = want.nbytes
    size = GUARD + 4096 + n + GUARD
    if kind == "pinned":
        raw = torch.empty(size, dtype=torch.uint8, pin_memory=True).numpy()
    else:
        raw = np.empty(size, np.uint8)
    start = GUARD + (-(raw.ctypes.data + GUARD)) % 4096 + shift
    if start + n + 1024 > size:
        raw = np.empty(size + 4096, np.uint8)
        start = GUARD + (-(raw.ctypes.data + GUARD)) % 4096 + shift
    if kind == "registered":
        assert int(torch.cuda.cudart().cudaHostRegister(raw.ctypes.data, raw.nbytes, 0)) == 0
    try:
        raw[:start] = 0xA5
        raw[start + n:] = 0xA5
        sess.reset()
        lumi_b200.api.check(lumi_b200.lib().lumi_prefill(sess._h, prompts[:batch].ctypes.data, batch, prompts.shape[1], C.c_void_p(raw.ctypes.data + start)))
        assert raw[start:start + n].tobytes() == want.tobytes()
        assert (raw[:start] == 0xA5).all() and (raw[start + n:] == 0xA5).all()
    finally:
        if kind == "registered":
            assert int(torch.cuda.cudart().cudaHostUnregister(raw.ctypes.data)) == 0
