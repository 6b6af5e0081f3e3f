"""GPU: waits of the product of prompt rows that run out (operands that the host has the kernel never request): the kernel ends, the call says so, and the next
products are right, also where K is split and CTAs of the same tile found the status set before they began."""
import pytest

import lumi_b200
from test_gpu_row_products import operands, product

pytestmark = pytest.mark.gpu


def run(a, w, d, skip, status):
    import torch
    torch.cuda.synchronize()
    return lumi_b200.lib().lumi_debug_row_gemm_wait_timeout(a.data_ptr(), w.data_ptr(), int(w.dtype == torch.bfloat16), d.data_ptr(), a.shape[0], w.shape[0], a.shape[1],
                                                            skip, status.data_ptr() if status is not None else 0)


# one tile; K in one piece over several tiles; K over three CTAs per tile and 228 CTAs: with 148 that are not fed, a tile's last share begins after the
# status is set (tiles of 64 and of 32 rows)
CASES = [(1, 1, 16, 1), (100, 300, 272, 2), (64, 9728, 1536, 148), (32, 9728, 1536, 148), (128, 5120, 1536, 1), (64, 9728, 1536, 1)]


@pytest.mark.parametrize("wdt", ["f32", "bf16"])
@pytest.mark.parametrize("M,N,K,skip", CASES)
def test_the_next_product_is_right(M, N, K, skip, wdt):
    import torch
    a, w = operands(M, N, K, wdt)
    other = -2 * a                                            # partial sums of the lost product are no help to the next one
    want = product(other, w)
    d = torch.zeros((M, N), device="cuda")
    product(a, w)
    status = torch.zeros(1, dtype=torch.int32, device="cuda")
    assert run(a, w, d, skip, status) == -7
    assert "wait expired" in lumi_b200.lib().lumi_last_error().decode()
    assert int(status.item()) == 4
    for _ in range(2):
        status.zero_()
        assert run(other, w, d.fill_(7.0), 0, status) == 0 and int(status.item()) == 0
        assert torch.equal(d, want)
        assert torch.equal(product(a, w), want / -2)


@pytest.mark.parametrize("M,N,K,skip", CASES)
def test_a_lost_wait_costs_time_and_no_result(M, N, K, skip):
    """Without a status word every CTA goes on, and what the tensor core did not deliver is summed by multiply-adds: the bound of the ordinary product."""
    import torch
    a, w = operands(M, N, K)
    want = product(a, w)
    ref = a.double() @ w.double().T
    product(-2 * a, w)                                        # partial sums of another product in the scratch memory
    d = torch.full((M, N), 7.0, device="cuda")
    assert run(a, w, d, skip, None) == 0
    assert (d.double() - ref).abs().max() < 2e-6 * ref.abs().max()
    product(-2 * a, w)
    assert torch.equal(product(a, w), want)
