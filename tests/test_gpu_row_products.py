"""GPU: the fp32 product of prompt rows (`lumi_k_row_gemm`): its results, its error against 64 bits and the order of its sums."""
import pytest

import lumi_b200

pytestmark = pytest.mark.gpu


def product(a, w, prev=None):
    import torch
    (M, K), N = a.shape, w.shape[0]
    d = torch.full((M, N), 7.0, device="cuda") if prev is None else prev.clone()
    torch.cuda.synchronize()
    lumi_b200.api.check(lumi_b200.lib().lumi_k_row_gemm(a.data_ptr(), w.data_ptr(), 1 if w.dtype == torch.bfloat16 else 0, d.data_ptr(), M, N, K, int(prev is not None), 0))
    torch.cuda.synchronize()
    return d


def operands(M, N, K, wdt="f32"):
    import torch
    g = torch.Generator(device="cuda").manual_seed(M + 3 * N + K)
    w = torch.randn((N, K), generator=g, device="cuda") * 0.05
    return torch.randn((M, K), generator=g, device="cuda"), w.to(torch.bfloat16) if wdt == "bf16" else w


WEIGHTS = ["f32", "bf16"]


# edges: tiles of 32 and 64 rows and 64 columns; K of one block, of an odd count, of less than a unit of 128, of a short last unit; K split and in one piece
@pytest.mark.parametrize("wdt", WEIGHTS)
@pytest.mark.parametrize("M,N,K", [(1, 1, 16), (4, 65, 48), (31, 64, 112), (32, 129, 128), (33, 100, 144), (64, 64, 1040), (65, 7, 272), (96, 1000, 320),
                                   (97, 520, 1024), (300, 1026, 2048), (8, 4100, 4096), (1000, 8200, 64)])
def test_matches_fp64(M, N, K, wdt):
    import torch
    a, w = operands(M, N, K, wdt)
    ref = a.double() @ w.double().T
    assert (product(a, w).double() - ref).abs().max() < 2e-6 * ref.abs().max()      # as for the streaming kernel
    prev = torch.randn((M, N), device="cuda")
    want = ref + prev.double()
    assert (product(a, w, prev).double() - want).abs().max() < 2e-6 * want.abs().max()


@pytest.mark.parametrize("wdt", WEIGHTS)
@pytest.mark.parametrize("K", [1024, 2048, 2816])
def test_no_further_from_64_bits_than_the_streaming_kernel(K, wdt):
    """A prompt must not lose bits by being taken a layer at a time: the same products by both kernels, 300 000 results.  An addition costs the square of
    its running sum; the kernel's order (chains of 16, units of four, groups of four) comes to 15.0 K of them at K = 1024 and 16.3 K at 2048, the
    streaming kernel's (at most chains of 16, five levels of a tree, segments of 512) to 14.5 K and 15.8 K: a ratio of errors of at most 1.02."""
    import torch
    M, N = 64, 4800
    a, w = operands(M, N, K, wdt)
    ref = a.double() @ w.double().T
    d = torch.empty((M, N), device="cuda")
    torch.cuda.synchronize()
    for m in range(0, M, 4):
        lumi_b200.api.check(lumi_b200.lib().lumi_k_gemv(a[m:].data_ptr(), w.data_ptr(), 1 if wdt == "bf16" else 0, d[m:].data_ptr(), 0, 0, 4, N, K, 0))
    torch.cuda.synchronize()
    rows, stream = ((x.double() - ref).square().mean().sqrt().item() for x in (product(a, w), d))
    assert rows <= 1.03 * stream, (rows, stream)


@pytest.mark.parametrize("wdt", WEIGHTS)
@pytest.mark.parametrize("N,K", [(1024, 2048), (7360, 1024), (200, 272)])
def test_a_row_is_the_same_alone_and_among_others(N, K, wdt):
    """Tiles of 32 and of 64 rows, K split over many, few and no CTAs."""
    import torch
    a, w = operands(700, N, K, wdt)
    whole = product(a, w)
    for M in (1, 5, 32, 40, 90, 200):
        assert torch.equal(product(a[:M], w), whole[:M]), M
