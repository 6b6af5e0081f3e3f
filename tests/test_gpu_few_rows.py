"""GPU: the tensor-core product for few rows (weights on the MMA's 128-row side, K shared by a cluster) at the edges of its tiles."""
import pytest

import lumi_b200

pytestmark = pytest.mark.gpu


# edges: rows 32 / 64 / 128 (padded rows of a tile) and two row tiles; weight rows 128; K of one k-block, of fewer than the stages, of
# uneven shares; N without whole quads, leading dimensions that forbid 16-byte access
@pytest.mark.parametrize("split", [True, False])
@pytest.mark.parametrize("M,N,K,ldd", [(1, 128, 64, 128), (9, 1, 64, 1), (31, 127, 128, 127), (32, 129, 192, 132), (33, 259, 1024, 259),
                                       (63, 1024, 2048, 1024), (64, 7360, 1024, 7360), (65, 1000, 4096, 1004), (127, 520, 320, 521),
                                       (128, 2048, 5632, 2048), (129, 1024, 2048, 1024), (300, 1026, 2112, 1028), (1024, 1024, 1024, 1024),
                                       (40, 40000, 128, 40000)])
def test_matches_fp64(split, M, N, K, ldd):
    import torch
    g = torch.Generator().manual_seed(M * 7 + N + K)
    a = torch.randn((M, K), generator=g)
    w = (torch.randn((N, K), generator=g) * 0.05).to(torch.bfloat16)
    hi = a.to(torch.bfloat16)
    lo = (a - hi.float()).to(torch.bfloat16)
    prev = torch.randn((M, ldd), generator=g)
    ref = ((hi.double() + lo.double()) if split else hi.double()) @ w.double().T
    hid, lod, wd = hi.cuda(), lo.cuda(), w.cuda()
    for acc in (0, 1):
        outs = []
        for _ in range(2):
            d = prev.clone().cuda()
            torch.cuda.synchronize()
            lumi_b200.api.check(lumi_b200.lib().lumi_k_gemm_bf16_tcgen05(hid.data_ptr(), lod.data_ptr() if split else 0, wd.data_ptr(), d.data_ptr(),
                                                                     M, N, K, ldd, acc, 0))
            torch.cuda.synchronize()
            outs.append(d.cpu())
        assert torch.equal(outs[0], outs[1])               # partial sums are added in split order
        want = ref + (prev[:, :N].double() if acc else 0)
        # products of bf16 are exact in fp32 and up to K of them are added with a rounding (or truncation) of 2^-23 of the running sum each;
        # such errors add up like a random walk: 2e-5 of the largest result is ten times what K = 5632 gives
        assert (outs[0][:, :N].double() - want).abs().max() < 2e-5 * want.abs().max()
        assert torch.equal(outs[0][:, N:], prev[:, N:])    # nothing beyond the last column is written


def test_a_wait_that_runs_out_is_reported():
    """One CTA's operands never arrive: its cluster still ends, the call answers with the timeout, and the next product is right."""
    import torch
    L = lumi_b200.lib()
    M, N, K = 64, 512, 1024
    g = torch.Generator(device="cuda").manual_seed(3)
    a = torch.randn((M, K), generator=g, device="cuda").to(torch.bfloat16)
    w = torch.randn((N, K), generator=g, device="cuda").to(torch.bfloat16)
    d = torch.zeros((M, N), device="cuda")
    ref = a.float() @ w.float().t()
    for skip, want in ((1, -7), (-1, 0)):
        status = torch.zeros(1, dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        assert L.lumi_debug_gemm_wait_timeout(a.data_ptr(), w.data_ptr(), d.data_ptr(), M, N, K, 2_000_000, skip, status.data_ptr()) == want
        assert bool(int(status.item()) & 4) == (want != 0)
    assert float((d - ref).abs().max() / ref.abs().max()) < 1e-5
