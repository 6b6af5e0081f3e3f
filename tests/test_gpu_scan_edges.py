"""The chunked prefill scan alone (lumi_k_ssd_prefill) against the recurrence in 64 bits, token by token (inference/src/model.rs:296-375):
lengths around its segments of 16 and chunks of 64 tokens, decays from almost none to total, and a neighbour's rows that are no numbers."""
import numpy as np
import pytest

import lumi_b200

P, N = 32, 64


def _recurrence(proj, st, w, H, G):
    """proj [T, R] of one sequence, st = (h, xprev, bprev, cum): gated outputs [T, H P] and the state behind them."""
    DI, BC = H * P, G * N
    h, xp, bp, cum = (a.astype(np.float64) for a in st)
    sig = lambda v: 1 / (1 + np.exp(-v))  # noqa: E731
    out = []
    for r in proj.astype(np.float64):
        x, z, b, c, dt, lam, dda, th = np.split(r, np.cumsum([DI, DI, BC, BC, H, H, H]))
        x, z = (x * sig(x)).reshape(H, P), z * sig(z)
        norm = lambda v, g, s: v / np.sqrt((v * v).mean() + 1e-5) * g + s  # noqa: E731
        b, c = (np.repeat(norm(v, w[g], w[s]).reshape(G, N), H // G, 0) for v, g, s in ((b, "bg", "bb"), (c, "cg", "cb")))
        dt = np.logaddexp(0, dt + w["dtb"])
        a = np.exp(np.clip(-np.logaddexp(0, dda), -1e6, -1e-4) * dt)
        lam = sig(lam)
        cum = cum + dt[:, None] * np.tanh(th.reshape(H, N // 2)) * np.float64(np.float32(np.pi))
        turn = lambda v: np.stack([v[:, 0::2] * np.cos(cum) - v[:, 1::2] * np.sin(cum), v[:, 0::2] * np.sin(cum) + v[:, 1::2] * np.cos(cum)], -1).reshape(H, N)  # noqa: E731
        b, c = turn(b), turn(c)
        u = lambda q, s: q[:, :, None] * s[:, None, :]  # noqa: E731
        h = a[:, None, None] * h + ((1 - lam) * a)[:, None, None] * u(xp, bp) + lam[:, None, None] * u(x, b)
        xp, bp = x, b
        y = (h * c[:, None, :]).sum(-1) + w["d"][:, None] * x
        out.append(y.reshape(-1) * z)
    return np.array(out), (h, xp, bp, cum)


@pytest.mark.gpu
@pytest.mark.parametrize("decay", [-3.0, 1.0, 60.0])
@pytest.mark.parametrize("T", [1, 15, 16, 17, 63, 64, 65, 200])
def test_scan_equals_the_recurrence(T, decay):
    import torch
    H, G, B = 8, 2, 2
    DI, BC = H * P, G * N
    R = 2 * DI + 2 * BC + 3 * H + H * N // 2
    g = np.random.default_rng(1000 * T + int(decay))
    proj = g.standard_normal((B, T, R)).astype(np.float32)
    o = 2 * DI + 2 * BC
    proj[:, :, o + 2 * H:o + 3 * H] += decay                     # e^(-60) per unit of dt: nothing is left of a token after the next
    w = {k: (1 + 0.1 * g.standard_normal(BC)).astype(np.float32) for k in ("bg", "cg", "bb", "cb")}
    w["d"] = (1 + 0.1 * g.standard_normal(H)).astype(np.float32)
    w["dtb"] = g.uniform(-2, 1, H).astype(np.float32)
    st = [g.standard_normal(s).astype(np.float32) for s in ((B, H, P, N), (B, H, P), (B, H, N), (B, H, N // 2))]
    proj[1] = np.nan                                             # boxes of the first sequence's last chunk reach into these rows
    dev = [torch.from_numpy(a).cuda() for a in st]
    params = [torch.from_numpy(w[k]).cuda() for k in ("bg", "cg", "bb", "cb", "d", "dtb")]
    rows = torch.from_numpy(proj.reshape(B * T, R)).cuda()
    yhi = torch.zeros((B * T, DI), dtype=torch.bfloat16, device="cuda")
    ylo, scratch = torch.zeros_like(yhi), torch.zeros(2 * B * T, dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    lumi_b200.api.check(lumi_b200.lib().lumi_k_ssd_prefill(rows.data_ptr(), R, *[p.data_ptr() for p in params], *[t.data_ptr() for t in dev],
                                                           yhi.data_ptr(), ylo.data_ptr(), scratch.data_ptr(), B, T, H, G, 0))
    torch.cuda.synchronize()
    got = (yhi.double() + ylo.double()).cpu().numpy().reshape(B, T, DI)[0]
    want, (h, xp, bp, cum) = _recurrence(proj[0], [a[0] for a in st], w, H, G)
    # both factors of every product are bf16 hi + lo (2^-17 each, lo lo left out: 2^-16), so a result is off by at most 2^-14 of the sum of
    # its terms' magnitudes; that sum is up to about 12 times the largest result here (64 terms of random sign, N = 64)
    assert np.abs(got - want).max() <= 12 * 2.0 ** -14 * np.abs(want).max()
    back = [t.cpu().numpy()[0].astype(np.float64) for t in dev]
    # angles are sums of up to T fp32 terms below 3 dt; they turn pairs of the state, so they are taken into its frame first
    off = back[3] - cum
    off -= 2 * np.pi * np.rint(off / (2 * np.pi))
    assert np.abs(off).max() < 1e-5 * (T + 8)
    turn = lambda v: np.stack([v[..., 0::2] * np.cos(o_) - v[..., 1::2] * np.sin(o_), v[..., 0::2] * np.sin(o_) + v[..., 1::2] * np.cos(o_)], -1).reshape(v.shape)  # noqa: E731
    o_ = off[:, None, :]
    assert np.abs(back[0] - turn(h)).max() <= 12 * 2.0 ** -14 * np.abs(h).max()
    o_ = off
    assert np.abs(back[2] - turn(bp)).max() <= 1e-5 * np.abs(bp).max() + 1e-5 * (T + 8) * 0.1
    assert np.abs(back[1] - xp).max() <= 1e-5 * np.abs(xp).max()
