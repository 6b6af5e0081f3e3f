"""GPU: every value of the gate of an attention block's MLP, alone, at widths that fill its blocks of two quads per thread or not."""
import pytest

import lumi_b200

pytestmark = pytest.mark.gpu


# 2, 258, 514 and 704 quads: one block of one warp, two quads a thread in one block, two blocks, two equal blocks; 512 quads fill one block
@pytest.mark.parametrize("width", [8, 1032, 2048, 2056, 2816])
@pytest.mark.parametrize("rows,pad", [(1, 0), (37, 4)])
def test_every_value(width, rows, pad):
    import torch
    g = torch.Generator(device="cuda").manual_seed(width + rows)
    ld = 2 * width + pad
    gu = torch.randn((rows, ld), generator=g, device="cuda") * 3
    gu[0, :4] = torch.tensor([100.0, -100.0, 0.0, -30.0])
    want = torch.sigmoid(gu[:, :width].double()) * gu[:, width:2 * width].double()
    for forms in ("f", "h", "hl", "fhl"):
        outs = {"f": torch.full((rows + 1, width), 7.0, device="cuda"),
                **{k: torch.full((rows + 1, width), 7.0, dtype=torch.bfloat16, device="cuda") for k in "hl"}}
        torch.cuda.synchronize()
        lumi_b200.api.check(lumi_b200.lib().lumi_k_gate_mul(gu.data_ptr(), ld, *(outs[k].data_ptr() if k in forms else 0 for k in "fhl"), rows, width, 0))
        torch.cuda.synchronize()
        for k, t in outs.items():
            assert bool((t[rows if k in forms else 0:] == 7.0).all()), (forms, k)      # the row behind the last, and what was not asked for
        size = want.abs()
        if "f" in forms:
            # exponential, sum, quotient and product: 2^-24 each, the exponential's 2 units in the last place
            assert bool(((outs["f"][:rows].double() - want).abs() <= 6 * 2.0 ** -24 * size + 1e-37).all())
        if "h" in forms:
            halves = outs["h"][:rows].double() + (outs["l"][:rows].double() if "l" in forms else 0)
            assert bool(((halves - want).abs() <= ((2.0 ** -16 if "l" in forms else 2.0 ** -8) + 6 * 2.0 ** -24) * size + 1e-37).all()), forms
