"""GPU: the fp32 product of prompt rows where its operands have one sign, so that what the tensor core cuts off of every sum adds up instead of averaging out; and
sums that lose nothing, which stay exact."""
import pytest

from test_gpu_row_products import product

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("wdt", ["f32", "bf16"])
@pytest.mark.parametrize("mean", [None, 2.0])
@pytest.mark.parametrize("K", [1024, 2048, 2816])
def test_as_close_to_64_bits_as_rounded_sums(K, mean, wdt):
    """The root mean square of 300 000 errors.  A rounded addition is off by at most 2^-24 / sqrt(3) of its result in the mean; the additions of one result, sized by
    their share of K: pairs of groups in order, a group to each pair's other, four k-blocks and the small products to a group (2.2 of its size squared), and
    the cut in each accumulator of 32.  1e-8 for what is not put back of the average cut."""
    import torch
    g = torch.Generator(device="cuda").manual_seed(K)
    a, w = torch.randn((64, K), generator=g, device="cuda"), torch.randn((4800, K), generator=g, device="cuda") * 0.05
    a, w = (a.abs(), w.abs()) if mean is None else (a + mean, w + 0.05 * mean)
    if wdt == "bf16":
        w = w.to(torch.bfloat16)
    ref = a.double() @ w.double().T
    err = (product(a, w).double() - ref) / ref.square().mean().sqrt()
    pairs = -(-K // 512)
    sizes = sum((k / pairs) ** 2 for k in range(2, pairs + 1)) + 1 / pairs + 2.2 * 256 / K + 32 / K
    assert err.square().mean().item() <= (2.0 ** -24) ** 2 / 3 * sizes + 1e-16
    assert abs(err.mean().item()) < 1.3e-8


# whole numbers whose sums stay below 2^21, and rows with a single entry: nothing is cut off, so nothing may be put back
@pytest.mark.parametrize("K", [16, 240, 2048])
def test_exact_sums_stay_exact(K):
    import torch
    g = torch.Generator(device="cuda").manual_seed(K)
    a, w = torch.randint(-20, 21, (40, K), generator=g, device="cuda").float(), torch.randint(-20, 21, (260, K), generator=g, device="cuda").float()
    assert torch.equal(product(a, w).double(), a.double() @ w.double().T)
    one = torch.zeros(40, K, device="cuda")
    at = torch.arange(40, device="cuda") * 7 % K
    one[torch.arange(40, device="cuda"), at] = 1.0
    w = torch.randn((260, K), generator=g, device="cuda") * torch.exp2(torch.randint(-20, 21, (260, K), generator=g, device="cuda").float())
    assert torch.equal(product(one, w), w.T[at])
