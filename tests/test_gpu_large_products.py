"""GPU: products whose work units go through several turns of a worker: pairs of CTAs over blocks of row tiles, streaming CTAs over groups
of weight rows."""
import pytest

import lumi_b200

pytestmark = pytest.mark.gpu


# edges: the first row count of the pairs, half-empty last row tiles and blocks, columns of one and of several widths, one k-block
@pytest.mark.parametrize("M,N,K,ldd", [(4096, 128, 64, 128), (4097, 260, 128, 260), (4300, 1000, 320, 1004), (8200, 520, 192, 520), (12289, 1024, 64, 1024),
                                       (4224, 4101, 128, 4101)])
def test_pairs_of_ctas_match_fp64(M, N, K, ldd):
    import torch
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    a = torch.randn((M, K), generator=g, device="cuda")
    w = (torch.randn((N, K), generator=g, device="cuda") * 0.05).to(torch.bfloat16)
    hi = a.to(torch.bfloat16)
    lo = (a - hi.float()).to(torch.bfloat16)
    prev = torch.randn((M, ldd), generator=g, device="cuda")
    ref = (hi.double() + lo.double()) @ w.double().T
    for acc in (0, 1):
        d = prev.clone()
        torch.cuda.synchronize()
        lumi_b200.api.check(lumi_b200.lib().lumi_k_gemm_bf16_tcgen05(hi.data_ptr(), lo.data_ptr(), w.data_ptr(), d.data_ptr(), M, N, K, ldd, acc, 0))
        torch.cuda.synchronize()
        want = ref + (prev[:, :N].double() if acc else 0)
        # exact products, up to 2 K = 640 additions of 2^-23 of the running sum each, as a random walk: 2e-5 of the largest result has room for ten times that
        assert (d[:, :N].double() - want).abs().max() < 2e-5 * want.abs().max()
        assert torch.equal(d[:, N:], prev[:, N:])


@pytest.mark.parametrize("wdt", ["f32", "bf16"])
@pytest.mark.parametrize("M,N,K", [(8, 20001, 1024), (5, 9473, 2048), (6, 4737, 4096), (3, 40007, 256), (1, 30011, 1024), (11, 9500, 128)])
def test_streaming_ctas_with_several_groups_of_rows(wdt, M, N, K):
    import torch
    g = torch.Generator(device="cuda").manual_seed(M + N + K)
    a = torch.randn((M, K), generator=g, device="cuda")
    w = torch.randn((N, K), generator=g, device="cuda") * 0.05
    w = w.to(torch.bfloat16) if wdt == "bf16" else w
    gamma = 1 + 0.1 * torch.randn(K, generator=g, device="cuda")
    res = torch.randn((M, N), generator=g, device="cuda")
    d = torch.empty((M, N), device="cuda")
    torch.cuda.synchronize()
    lumi_b200.api.check(lumi_b200.lib().lumi_k_gemv(a.data_ptr(), w.data_ptr(), 1 if wdt == "bf16" else 0, d.data_ptr(), res.data_ptr(), gamma.data_ptr(),
                                                M, N, K, 0))
    torch.cuda.synchronize()
    x = a.double()
    x = x / torch.sqrt((x * x).mean(1, keepdim=True) + 1e-5) * gamma.double()
    ref = x @ w.double().T + res.double()
    # fp32 throughout: lanes add K / 32 products each, then a tree; 2e-6 of the largest result as for the shorter products
    assert (d.double() - ref).abs().max() < 2e-6 * ref.abs().max()


def test_a_long_prompt_has_the_same_state_alone_and_among_others():
    """Alone its products have 1024 rows (single CTAs), among 31 others 32768 (pairs of CTAs, blocks of row tiles): the sums run in one order."""
    import numpy as np
    from lumi_b200 import synth
    cfg = synth.base_config(n_layers=3, vocab_size=500, attention_layers=[1], attn_mlp_dim=256, attn_rope_base=10000.0)
    model = lumi_b200.NmModel.from_tensors(cfg, list(synth.iter_tensors(cfg, seed=29, weights_dtype="bf16", perturb_ones=0.05)))
    prompts = synth.random_prompts(32, 1024, cfg.vocab_size, seed=31)
    many, one = model.init_states(32, 1030), model.init_states(1, 1030)
    many.prefill(prompts, want_logits=False)
    for b in (0, 17, 31):
        one.reset()
        one.prefill(prompts[b:b + 1], want_logits=False)
        for layer in (0, 2):
            for x, y in zip(many.read_state(b, layer), one.read_state(0, layer)):
                assert np.array_equal(x, y), (b, layer)
