"""Several weights of different sizes in one SGD launch: each as if it were alone."""

import pytest
import torch

from moonep_b200.ops.moe_ops import sgd_update, sgd_updates


# one to seven weights (up to three launches), none, remainders of a CTA's elements, one that is no multiple of eight
SIZES = [[8], [2056, 8], [0, 2048, 148 * 8 * 2048 + 8], [8, 0, 0], [64, 12, 4096], [8, 16, 24, 32, 40, 48, 56], []]


@pytest.mark.parametrize("sizes", SIZES)
def test_updates_on_the_cpu(sizes):
    ws, gs = ([torch.arange(n).to(d) for n in sizes] for d in (torch.bfloat16, torch.float32))
    want = [w - 0.5 * g for w, g in zip([w.float() for w in ws], gs)]
    sgd_updates(ws, gs, 0.5)
    assert all(torch.equal(w, t.bfloat16()) for w, t in zip(ws, want))


@pytest.mark.gpu
@pytest.mark.parametrize("sizes", SIZES)
def test_updates_together_and_alone(sizes):
    g = torch.Generator(device="cuda").manual_seed(len(sizes))
    # spaced by eight elements that no update may touch
    whole = [torch.randn(n + 8, generator=g, device="cuda").bfloat16() for n in sizes]
    alone, gs = [w.clone() for w in whole], [torch.randn(n, generator=g, device="cuda") for n in sizes]
    sgd_updates([w[:-8] for w in whole], gs, 0.25)
    for w, gr in zip(alone, gs):
        sgd_update(w[:-8], gr, 0.25)
    assert all(torch.equal(a, b) for a, b in zip(whole, alone))


@pytest.mark.gpu
def test_update_of_a_view_that_is_not_aligned():
    w, gr = torch.randn(17, device="cuda").bfloat16(), torch.randn(18, device="cuda")
    want = w[1:].double() - 0.25 * gr[2:].double()
    sgd_updates([w[1:]], [gr[2:]], 0.25)
    # the product is exact, the difference rounded to fp32 and to bf16
    assert bool(((w[1:].double() - want).abs() <= (2.0**-8 + 2.0**-23) * want.abs()).all())
