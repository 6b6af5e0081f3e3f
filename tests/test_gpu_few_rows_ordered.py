"""GPU: the kernel for products of few rows in its ordered form gives the bits of the persistent kernel, with every epilogue that models with experts ask for."""
import pytest

from test_gpu_product_epilogues import Case

pytestmark = pytest.mark.gpu
FORMS = {"ordered": dict(few_rows=1, ordered=1), "split": {}}      # over the persistent kernel with a split of K


def halves_of(M, N):
    import torch
    return [torch.zeros(M, N, dtype=torch.bfloat16, device="cuda") for _ in range(2)]


# K in one piece, shared by two and by four CTAs; rows of every tile height; above 64 rows only what is shared goes there
@pytest.mark.parametrize("M", [1, 23, 33, 64, 100, 128])
@pytest.mark.parametrize("N,K", [(32, 64), (2048, 2048), (2048, 5632), (1024, 1408), (4096, 1024), (1024, 2816), (1056, 1024)])
def test_same_bits(M, N, K):
    import torch
    c = Case(M, N, K)
    ssq, bias, gamma, old = c.rand(M, 4).square() * K / 3, c.rand(N), 1 + 0.1 * c.rand(N), c.rand(M, N)
    got = {}
    for form, kernel in FORMS.items():
        out = got[form] = []
        d = torch.zeros(M, N, device="cuda")
        c.run("split", **kernel, d=d, ssq_in=ssq, ssq_parts=3, ssq_stride=4, inv_k=1.0 / K, eps=1e-5)
        out.append(d)
        hi, lo = halves_of(M, N)
        c.run("split", **kernel, act=2, out_hi=hi, out_lo=lo)
        out += [hi, lo]
        for b in ({}, dict(bias=bias)):
            d, (hi, lo), sums = old.clone(), halves_of(M, N), torch.zeros(M, N // 32, device="cuda")
            c.run("split", **kernel, d=d, accumulate=1, gamma_next=gamma, out_hi=hi, out_lo=lo, ssq_out=sums, ssq_stride=N // 32, **b)
            out += [d, hi, lo, sums]
    for i, (a, b) in enumerate(zip(got["ordered"], got["split"])):
        assert torch.equal(a, b), i


@pytest.mark.parametrize("M", [1, 23, 64])
@pytest.mark.parametrize("groups,group_rows,out_n,K", [(1, 5632, 5632, 1024), (8, 256, 256, 128), (5, 160, 157, 192), (16, 96, 90, 320)])
def test_same_bits_in_groups(M, groups, group_rows, out_n, K):
    import torch
    c = Case(M, groups * group_rows, K, groups)
    n = groups * out_n
    bias, mul, ssq = c.rand(groups * group_rows), c.rand(M, n), c.rand(M, 4).square() * K / 3
    shape = dict(groups=groups, group_rows=group_rows, lda=groups * K)
    got = {}
    for form, kernel in FORMS.items():
        out = got[form] = []
        for kw in ({}, dict(bias=bias), dict(bias=bias, mul=mul, ldmul=n)):
            d, (hi, lo) = torch.zeros(M, n, device="cuda"), halves_of(M, n)
            c.run("split", **kernel, d=d, ldd=n, out_hi=hi, out_lo=lo, ldo=n, out_step=out_n, out_n=out_n, **kw, **shape)
            out += [d, hi, lo]
        if groups == 1:
            for gate in (3, 4):
                for kw in ({}, dict(bias=bias)):
                    hi, lo = halves_of(M, out_n // 2)
                    c.run("split", **kernel, out_hi=hi, out_lo=lo, ldo=out_n // 2, out_step=out_n // 2, out_n=out_n // 2, gate=gate, ssq_in=ssq, ssq_parts=3, ssq_stride=4,
                          inv_k=1.0 / K, eps=1e-5, **kw, **shape)
                    out += [hi, lo]
    for i, (a, b) in enumerate(zip(got["ordered"], got["split"])):
        assert torch.equal(a, b), i
