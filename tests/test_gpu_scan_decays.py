"""GPU: the chunked prefill scan alone where a token lets next to nothing through of what came before it and the tokens around it nearly everything: the decays
behind such a token must not suffer from it.  Against the recurrence in 64 bits, token by token (inference/src/model.rs:296-375)."""
import numpy as np
import pytest

import lumi_b200
from test_gpu_scan_edges import N, P, _recurrence

pytestmark = pytest.mark.gpu


# places of the strong tokens in segments of 16: the first and second of a pair, the last of a segment, neighbours, none in a whole segment, all of one
@pytest.mark.parametrize("strong", [1e6, 400.0, 90.0, 30.0])
@pytest.mark.parametrize("places", [[1], [0, 17, 35], [5, 6, 7, 15, 16, 47], list(range(16, 32)), [2, 9, 63, 64, 100]])
def test_decays_behind_a_total_one(places, strong):
    import torch
    H, G, T = 8, 2, 130
    DI, BC = H * P, G * N
    o = 2 * DI + 2 * BC
    R = o + 3 * H + H * N // 2
    g = np.random.default_rng(int(strong) + len(places))
    proj = g.standard_normal((1, T, R)).astype(np.float32)
    proj[:, :, o:o + H] = 1.0 + 0.1 * proj[:, :, o:o + H]          # dt about 1
    proj[:, :, o + 2 * H:o + 3 * H] = -4.0                          # a token lets 0.98 through
    proj[:, places, o + 2 * H:o + 3 * H] = strong                   # e^(-strong)
    w = {k: (1 + 0.1 * g.standard_normal(BC)).astype(np.float32) for k in ("bg", "cg", "bb", "cb")}
    w["d"] = (1 + 0.1 * g.standard_normal(H)).astype(np.float32)
    w["dtb"] = g.uniform(-0.2, 0.2, H).astype(np.float32)
    st = [g.standard_normal(s).astype(np.float32) for s in ((1, H, P, N), (1, H, P), (1, H, N), (1, H, N // 2))]
    want, (h, _, _, cum) = _recurrence(proj[0], [a[0] for a in st], w, H, G)
    dev = [torch.from_numpy(a).cuda() for a in st]
    params = [torch.from_numpy(w[k]).cuda() for k in ("bg", "cg", "bb", "cb", "d", "dtb")]
    rows = torch.from_numpy(proj.reshape(T, R)).cuda()
    yhi = torch.zeros((T, DI), dtype=torch.bfloat16, device="cuda")
    ylo, scratch = torch.zeros_like(yhi), torch.zeros(2 * T, dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    lumi_b200.api.check(lumi_b200.lib().lumi_k_ssd_prefill(rows.data_ptr(), R, *[p.data_ptr() for p in params], *[t.data_ptr() for t in dev],
                                                           yhi.data_ptr(), ylo.data_ptr(), scratch.data_ptr(), 1, T, H, G, 0))
    torch.cuda.synchronize()
    got = (yhi.double() + ylo.double()).cpu().numpy()
    # as in the test of the edges: 2^-14 of the sum of a result's terms, which is up to about 12 times the largest result here; logarithms count as -88 at
    # least, so behind the up to three strong tokens of a segment here a decay is off by 2^-15 of itself (four roundings of sums up to 264, 2^-17 each)
    assert np.abs(got - want).max() <= 12 * 2.0 ** -14 * np.abs(want).max()
    off = dev[3].cpu().numpy()[0].astype(np.float64) - cum
    off -= 2 * np.pi * np.rint(off / (2 * np.pi))
    s, c = np.sin(off)[:, None, :], np.cos(off)[:, None, :]
    turned = np.stack([h[..., 0::2] * c - h[..., 1::2] * s, h[..., 0::2] * s + h[..., 1::2] * c], -1).reshape(h.shape)
    assert np.abs(dev[0].cpu().numpy()[0] - turned).max() <= 12 * 2.0 ** -14 * np.abs(h).max()
