"""GPU: after a product with K split whose wait ran out the call leaves the tile counters at zero: the next product with another split is right.  (It does not write a tile
whose counter is beyond its own number of splits; with the same number, partial sums that arrive in time hide the fault.)"""
import ctypes as C

import pytest

import lumi_b200
from test_gpu_product_epilogues import Case

pytestmark = pytest.mark.gpu


def splits(c):
    w, s = C.c_int32(), C.c_int32()
    lumi_b200.api.check(lumi_b200.lib().lumi_debug_gemm_plan(c.M, c.N, c.K, 1, 0, C.byref(w), C.byref(s)))
    return s.value


@pytest.mark.parametrize("unit", [0, 1, 127])
def test_the_next_product_with_k_split_is_right(unit):
    import torch
    four, two = Case(64, 1024, 2048), Case(64, 3072, 4608)
    assert (splits(four), splits(two)) == (4, 2)
    want = [c.a64 @ c.w.double().T for c in (four, two)]
    lost, status = torch.zeros(64, 1024, device="cuda"), torch.zeros(1, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    p = four.probe("split", d=lost, status_word=status, wait_limit_ns=2_000_000, skip_unit=unit)
    assert lumi_b200.lib().lumi_debug_gemm(C.byref(p)) == -7
    # the status still set: a launch that does no work leaves them at zero, too
    p = two.probe("split", d=torch.zeros(64, 3072, device="cuda"), status_word=status, wait_limit_ns=2_000_000)
    assert lumi_b200.lib().lumi_debug_gemm(C.byref(p)) == -7
    for i in (1, 0, 1):
        c = (four, two)[i]
        d = torch.full((64, c.N), 7.0, device="cuda")
        c.run("split", d=d)
        assert float((d.double() - want[i]).abs().max()) < 2e-5 * float(want[i].abs().max())      # as in the tests of the epilogues
