"""GPU: every kernel that takes the steps' tensor-core products (the one for few rows, single CTAs with and without a split of K, pairs of CTAs), each with
the epilogues that a step asks of it, at the edges of tiles; which of them give the same bits; and waits that run out."""
import ctypes as C

import pytest

import lumi_b200
from lumi_b200.api import GemmProbe

pytestmark = pytest.mark.gpu

KERNELS = {"few": dict(few_rows=1), "single": dict(), "split": dict(split_k=1), "pair": dict(pairs=1)}


class Case:
    """Operands of one product and its epilogue; fp64 references."""

    def __init__(self, M, N, K, groups=0, seed=0):
        import torch
        g = torch.Generator(device="cuda").manual_seed(seed + M + 3 * N + 7 * K)
        self.M, self.N, self.K = M, N, K
        self.rand = lambda *shape: torch.randn(shape, generator=g, device="cuda")
        a = self.rand(M, K * max(1, groups))
        self.hi = a.to(torch.bfloat16)
        self.lo = (a - self.hi.float()).to(torch.bfloat16)
        self.w = (self.rand(N, K) * 0.05).to(torch.bfloat16)
        self.a64 = self.hi.double() + self.lo.double()

    def probe(self, kernel, **kw):
        p = GemmProbe(M=self.M, N=self.N, K=self.K, ldd=self.N, a_hi=self.hi.data_ptr(), a_lo=self.lo.data_ptr(), w=self.w.data_ptr(), skip_unit=-1)
        for k, v in {**KERNELS[kernel], **kw}.items():
            setattr(p, k, v.data_ptr() if hasattr(v, "data_ptr") else v)
        return p

    def run(self, kernel, **kw):
        import torch
        torch.cuda.synchronize()
        p = self.probe(kernel, **kw)
        lumi_b200.api.check(lumi_b200.lib().lumi_debug_gemm(C.byref(p)))
        torch.cuda.synchronize()


def close(got, want):
    # exact products, at most 2 K additions of 2^-23 of the running sum each, as a random walk: 2e-5 of the largest result is ten times what K = 4096
    # gives; results as two bf16 halves add 2^-17 of their own size
    assert float((got.double() - want).abs().max()) < 2e-5 * float(want.abs().max())


def halves(hi, lo):
    return hi.double() + lo.double()


# few: tiles of 32 / 64 / 128 rows and 128 weight rows, K shared and not; split: K over two and four CTAs; pair: 256 rows, widths 128 / 192 / 256
SHAPES = [("few", 1, 8, 64), ("few", 33, 136, 192), ("few", 64, 1000, 1024), ("few", 127, 264, 320), ("few", 300, 1032, 2112),
          ("single", 33, 136, 192), ("single", 129, 1000, 320), ("single", 4097, 264, 128),
          ("split", 64, 1024, 2048), ("split", 100, 1024, 2816), ("split", 64, 1000, 2048), ("split", 128, 264, 4096), ("split", 17, 40, 1024),
          ("pair", 4096, 8, 64), ("pair", 4097, 264, 128), ("pair", 4300, 1000, 320), ("pair", 5000, 520, 192)]


@pytest.mark.parametrize("kernel,M,N,K", SHAPES)
def test_norm_folded_around_a_product(kernel, M, N, K):
    import torch
    c = Case(M, N, K)
    parts, stride, eps = 5, 8, 1e-5
    ssq = c.rand(M, stride).square() * K / parts
    scale = 1 / torch.sqrt(ssq[:, :parts].double().sum(1, keepdim=True) / K + eps)
    bias, gamma, old = c.rand(N), 1 + 0.1 * c.rand(N), c.rand(M, N)
    want = (c.a64 @ c.w.double().T) * scale + bias.double()
    consumer = dict(ssq_in=ssq, ssq_parts=parts, ssq_stride=stride, inv_k=1.0 / K, eps=eps, bias=bias)
    d = torch.full_like(old, 7.0)
    c.run(kernel, d=d, **consumer)
    close(d, want)
    # the residual stream: added to what is there, the next norm's input and sums of squares beside it
    d, hi, lo = old.clone(), torch.empty(M, N, dtype=torch.bfloat16, device="cuda"), torch.empty(M, N, dtype=torch.bfloat16, device="cuda")
    strips = (N + 31) // 32
    sums = torch.full((M, strips + 3), -1.0, device="cuda")
    c.run(kernel, d=d, accumulate=1, bias=bias, gamma_next=gamma, out_hi=hi, out_lo=lo, ssq_out=sums, ssq_stride=strips + 3)
    want = c.a64 @ c.w.double().T + bias.double() + old.double()
    close(d, want)
    close(halves(hi, lo), want * gamma.double())
    padded = torch.zeros(M, strips * 32, dtype=torch.float64, device="cuda")
    padded[:, :N] = want.square()
    want = padded.view(M, strips, 32).sum(2)
    assert float((sums[:, :strips].double() - want).abs().max()) < 1e-4 * float(want.max())
    assert bool((sums[:, strips:] == -1.0).all())


@pytest.mark.parametrize("kernel,M,N,K", SHAPES)
def test_activation_into_halves(kernel, M, N, K):
    import torch
    c = Case(M, N, K)
    hi, lo = torch.empty(M, N, dtype=torch.bfloat16, device="cuda"), torch.empty(M, N, dtype=torch.bfloat16, device="cuda")
    c.run(kernel, act=2, out_hi=hi, out_lo=lo)
    close(halves(hi, lo), torch.relu(c.a64 @ c.w.double().T).square())


# groups of weight rows that are no whole tiles, results narrower than the group, outputs that forbid wide stores
@pytest.mark.parametrize("kernel", ["few", "single"])
@pytest.mark.parametrize("M,groups,group_rows,out_n,K", [(1, 1, 32, 32, 64), (33, 3, 96, 90, 64), (64, 5, 160, 157, 192), (130, 2, 128, 128, 1024)])
def test_products_in_groups(kernel, M, groups, group_rows, out_n, K):
    import torch
    c = Case(M, groups * group_rows, K, groups)
    n = groups * out_n
    bias, mul = c.rand(groups * group_rows), c.rand(M, n)
    want = torch.cat([c.a64[:, g * K:(g + 1) * K] @ c.w[g * group_rows:g * group_rows + out_n].double().T + bias[g * group_rows:g * group_rows + out_n].double()
                      for g in range(groups)], 1) * torch.sigmoid(mul.double())
    d, hi, lo = torch.full((M, n + 2), 7.0, device="cuda"), *(torch.zeros(M, n, dtype=torch.bfloat16, device="cuda") for _ in range(2))
    c.run(kernel, d=d, ldd=n + 2, bias=bias, mul=mul, ldmul=n, out_hi=hi, out_lo=lo, ldo=n, groups=groups, group_rows=group_rows, lda=groups * K, out_step=out_n,
          out_n=out_n)
    close(d[:, :n], want)
    close(halves(hi, lo), want)
    assert bool((d[:, n:] == 7.0).all())


@pytest.mark.parametrize("kernel", ["few", "single"])
@pytest.mark.parametrize("gate", [3, 4])
@pytest.mark.parametrize("M,N,K", [(9, 32, 64), (33, 160, 128), (64, 416, 1024), (300, 5632, 64)])
def test_gated_results(kernel, M, N, K, gate):
    import torch
    c = Case(M, N, K)
    parts = 3
    ssq = c.rand(M, 4).square() * K / parts
    scale = 1 / torch.sqrt(ssq[:, :parts].double().sum(1, keepdim=True) / K + 1e-5)
    v = ((c.a64 @ c.w.double().T) * scale).view(M, N // 32, 2, 16)
    g, up = v[:, :, 0].reshape(M, N // 2), v[:, :, 1].reshape(M, N // 2)
    want = (torch.relu(g) if gate == 3 else torch.nn.functional.silu(g)) * up
    hi, lo = (torch.empty(M, N // 2, dtype=torch.bfloat16, device="cuda") for _ in range(2))
    c.run(kernel, out_hi=hi, out_lo=lo, ldo=N // 2, groups=1, group_rows=N, lda=K, out_step=N // 2, out_n=N // 2, gate=gate, ssq_in=ssq, ssq_parts=parts,
          ssq_stride=4, inv_k=1.0 / K, eps=1e-5)
    close(halves(hi, lo), want)


@pytest.mark.parametrize("M,N,K", [(4096, 128, 64), (4300, 1024, 2048), (4097, 4101, 128), (8200, 1536, 1024), (5000, 2048, 5632)])
@pytest.mark.parametrize("accumulate", [0, 1])
def test_pairs_give_the_same_bits_as_single_ctas(M, N, K, accumulate):
    """What lets a sequence have the same state alone and among others, on either side of the row count from which pairs take the products."""
    import torch
    c = Case(M, N, K)
    outs = [torch.full((M, N), 0.3, device="cuda") for _ in range(3)]
    c.run("pair", d=outs[0], accumulate=accumulate)
    c.run("single", d=outs[1], accumulate=accumulate)
    assert torch.equal(outs[0], outs[1])
    few = 1000                                               # single CTAs with other tile widths
    c.M = few
    c.run("single", d=outs[2], accumulate=accumulate)
    assert torch.equal(outs[2][:few], outs[0][:few])


@pytest.mark.parametrize("kernel,M,N,K,unit", [("few", 64, 512, 1024, 1), ("single", 4300, 512, 1024, 1), ("pair", 4300, 512, 1024, 1), ("pair", 4300, 512, 128, 33),
                                               ("pair", 40000, 512, 320, 100)])
def test_a_wait_that_runs_out_is_reported(kernel, M, N, K, unit):
    """Operands of one work unit never arrive (of a pair: the second CTA's, so that the first one's copies have nobody to be consumed with): the kernel ends,
    the call answers with the timeout, and the next product is right.  The last case stops in a worker's second unit."""
    import torch
    c = Case(M, N, K)
    d = torch.zeros(M, N, device="cuda")
    for skip, want in ((unit, -7), (-1, 0)):
        status = torch.zeros(1, dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        p = c.probe(kernel, d=d, status_word=status, wait_limit_ns=2_000_000, skip_unit=skip)
        assert lumi_b200.lib().lumi_debug_gemm(C.byref(p)) == want
        assert bool(int(status.item()) & 4) == (want != 0)
    close(d, c.a64 @ c.w.double().T)
