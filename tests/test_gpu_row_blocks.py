"""GPU: products over some blocks of 32 rows only (prompts of different lengths): the rows of the list have the bits that they have without it, the others
of the result stay what they were."""
import pytest

from test_gpu_product_epilogues import Case

pytestmark = pytest.mark.gpu


# the first and the last block (of fewer rows than 32), a single one, tiles that the list's end cuts; single CTAs and pairs (4096 listed rows and more)
@pytest.mark.parametrize("kernel,M,keep", [("single", 1030, [32]), ("single", 1500, [0, 3, 4, 5, 46]), ("single", 4000, 0.6), ("pair", 9000, 0.7), ("pair", 8193, 0.55)])
@pytest.mark.parametrize("form", ["residual", "norm", "gate", "groups"])
def test_listed_rows_only(kernel, M, keep, form):
    import torch
    N, K, groups = {"residual": (328, 192, 0), "norm": (1000, 128, 0), "gate": (416, 128, 0), "groups": (480, 64, 3)}[form]
    c = Case(M, N, K, groups)
    blocks = (M + 31) // 32
    if not isinstance(keep, list):
        pick = torch.randperm(blocks, generator=torch.Generator().manual_seed(M))[:int(keep * blocks)]
        keep = sorted({0, blocks - 1, *pick.tolist()})
    listed = torch.zeros(M, dtype=torch.bool, device="cuda")
    for b in keep:
        listed[32 * b:32 * b + 32] = True
    dev = torch.tensor(keep, dtype=torch.int32, device="cuda")
    ssq, bias, gamma, old = c.rand(M, 4).square() * K / 3, c.rand(N), 1 + 0.1 * c.rand(N), c.rand(M, N)
    consumer = dict(ssq_in=ssq, ssq_parts=3, ssq_stride=4, inv_k=1.0 / K, eps=1e-5)

    def outputs(**extra):
        n = {"gate": N // 2}.get(form, N)
        hi, lo = (torch.full((M, n), 3.0, dtype=torch.bfloat16, device="cuda") for _ in range(2))
        d, sums = old.clone(), torch.full((M, (N + 31) // 32), -1.0, device="cuda")
        if form == "residual":
            c.run(kernel, d=d, accumulate=1, bias=bias, gamma_next=gamma, out_hi=hi, out_lo=lo, ssq_out=sums, ssq_stride=sums.shape[1], **extra)
        elif form == "norm":
            c.run(kernel, d=d, bias=bias, **consumer, **extra)
        elif form == "gate":
            c.run(kernel, out_hi=hi, out_lo=lo, ldo=n, groups=1, group_rows=N, lda=K, out_step=n, out_n=n, gate=3, **consumer, **extra)
        else:
            c.run(kernel, d=d, bias=bias, groups=groups, group_rows=N // groups, lda=groups * K, out_step=N // groups, out_n=N // groups, **extra)
        return {"d": d, "hi": hi, "lo": lo, "sums": sums}

    every, some = outputs(), outputs(row_blocks=dev, n_row_blocks=len(keep))
    for k, v in some.items():
        assert torch.equal(v[listed], every[k][listed]), k
        before = {"d": old, "hi": torch.full_like(v, 3.0), "lo": torch.full_like(v, 3.0), "sums": torch.full_like(v, -1.0)}[k]
        assert torch.equal(v[~listed], before[~listed]), k
