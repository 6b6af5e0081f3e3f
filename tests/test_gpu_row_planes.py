"""GPU: the fp32 product of prompt rows where its three planes per operand are put to the test: numbers of very different sizes, rows that are no numbers, and
the edges of its tiles of 128 weight rows and of its groups of 256 of K."""
import pytest

from test_gpu_row_products import product

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("wdt", ["f32", "bf16"])
@pytest.mark.parametrize("M,N,K", [(1, 127, 16), (33, 128, 240), (64, 129, 256), (65, 255, 272), (32, 257, 2064)])
def test_every_bit_of_operands_of_any_size(M, N, K, wdt):
    """Sizes from 2^-30 to 2^30 side by side: an error is bounded by the sum of its terms' magnitudes.  The planes left out are 3 * 2^-25 of a term, at most
    two terms of 16 lose 2^-23 of a running sum each in an accumulator and the sums of accumulators 2^-24 a time, at most 32 + K / 32 times."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    rand = lambda *s: torch.randn(s, generator=g, device="cuda") * torch.exp2(torch.randint(-30, 31, s, generator=g, device="cuda").float())  # noqa: E731
    a, w = rand(M, K), rand(N, K)
    if wdt == "bf16":
        w = w.to(torch.bfloat16)
    ref, size = a.double() @ w.double().T, a.double().abs() @ w.double().abs().T
    assert bool(((product(a, w).double() - ref).abs() <= (2 + (32 + K / 32) / 2) * 2.0 ** -23 * size).all())


@pytest.mark.parametrize("wdt", ["f32", "bf16"])
def test_a_row_without_numbers_stays_alone(wdt):
    import torch
    g = torch.Generator(device="cuda").manual_seed(5)
    a, w = torch.randn((70, 528), generator=g, device="cuda"), torch.randn((300, 528), generator=g, device="cuda")
    if wdt == "bf16":
        w = w.to(torch.bfloat16)
    whole = product(a, w)
    a[7, 100], a[40, 3], a[69, 527] = float("inf"), float("nan"), -float("inf")
    got = product(a, w)
    bad = torch.zeros(70, dtype=torch.bool, device="cuda")
    bad[[7, 40, 69]] = True
    assert torch.equal(got[~bad], whole[~bad])
    assert not bool(torch.isfinite(got[bad]).any())
