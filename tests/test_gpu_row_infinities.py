"""GPU: the fp32 product of prompt rows with operands that have no three finite bf16 planes: infinities, and numbers above bf16's largest.  What multiply-adds
give: infinities of the right sign, finite results, and no number only where two infinities or an infinity and a zero meet."""
import pytest

from test_gpu_row_products import operands, product

pytestmark = pytest.mark.gpu
INF = float("inf")
BIG = 3.4e38                                                  # rounds to infinity in bf16


def check(a, w, touched, prev=None):
    import torch
    want = a.double() @ w.double().T                          # nothing overflows 64 bits: the infinities are those of the operands
    want = want if prev is None else want + prev.double()
    got = product(a, w, prev).double()
    assert torch.equal(torch.isnan(got), torch.isnan(want))
    assert torch.equal(got[want.isinf()], want[want.isinf()])
    fin = want.isfinite()
    size = a.double().abs().nan_to_num(0, 0, 0) @ w.double().abs().nan_to_num(0, 0, 0).T
    bound = (2 + (32 + a.shape[1] / 32) / 2) * 2.0 ** -23 * size      # as for finite operands of any size
    bound += 0 if prev is None else 2.0 ** -24 * want.abs()
    assert bool(((got - want).abs()[fin] <= bound[fin]).all())
    assert bool(fin.any()) and bool((want.isinf() | (want.abs() > 1e30))[touched].any())


# rows of whole tiles and of a tile's edge, K in one piece and split
@pytest.mark.parametrize("wdt", ["f32", "bf16"])
@pytest.mark.parametrize("M,N,K", [(70, 300, 528), (32, 129, 2048), (3, 1, 16)])
def test_activations(M, N, K, wdt):
    import torch
    a, w = operands(M, N, K, wdt)
    a[0, 3], a[1, K - 1], a[M - 1, 5] = INF, -INF, BIG
    w[0, 3] = 0                                               # infinity times zero
    if M > 40:
        a[37, 1], a[37, 200] = INF, -INF                      # no number for most columns
    touched = torch.arange(M, device="cuda") % (M - 1) <= 1
    check(a, w, touched)
    check(a, w, touched, torch.randn((M, N), device="cuda"))  # added to what is there


@pytest.mark.parametrize("wdt", ["f32", "bf16"])
@pytest.mark.parametrize("M,N,K", [(70, 300, 528), (32, 129, 2048)])
def test_weights(M, N, K, wdt):
    import torch
    a, w = operands(M, N, K, wdt)
    a[:, 2] *= 0.1                                            # the large products stay finite in 32 bits
    w[7, 100], w[N - 1, K - 1], w[8, 2] = INF, -INF, BIG if wdt == "f32" else 3.38e38
    check(a, w, torch.ones(M, dtype=torch.bool, device="cuda"))
