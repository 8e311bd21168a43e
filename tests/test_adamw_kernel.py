"""The one-pass AdamW kernel against the same step in 64 bits, at sizes around its vectors and grid."""

import pytest
import torch

from moonep_b200.ops.moe_ops import adamw_update


@pytest.mark.parametrize(
    "device,sizes,shift",
    [
        ("cpu", [12], 0),
        ("cpu", [], 0),
        ("cpu", [4, 8, 12, 16], 0),
        pytest.param("cuda", [4], 0, marks=pytest.mark.gpu),
        pytest.param("cuda", [1020, 1024, 1028], 0, marks=pytest.mark.gpu),
        pytest.param("cuda", [8, 4, 1024, 64, 1028, 16, 12], 0, marks=pytest.mark.gpu),  # three launches
        # just short of, at and past one vector per thread of a full GPU, then two and four of them
        pytest.param("cuda", [148 * 8 * 1024 - 4, 8], 0, marks=pytest.mark.gpu),
        pytest.param("cuda", [148 * 8 * 1024 + 4, 8], 0, marks=pytest.mark.gpu),
        pytest.param("cuda", [148 * 16 * 1024 + 4], 0, marks=pytest.mark.gpu),
        pytest.param("cuda", [148 * 40 * 1024 + 1028], 0, marks=pytest.mark.gpu),
        pytest.param("cuda", [1001, 64], 0, marks=pytest.mark.gpu),  # not whole vectors: elementwise operations
        pytest.param("cuda", [64, 64], 1, marks=pytest.mark.gpu),  # not 16-byte aligned: elementwise operations
    ],
)
def test_adamw_step(device, sizes, shift):
    g = torch.Generator(device=device).manual_seed(sum(sizes))

    def make(n, dtype=torch.float32):
        return torch.empty(n + shift, dtype=dtype, device=device)[shift:].copy_(torch.randn(n, generator=g, device=device))

    p, m, gr = ([make(n) for n in sizes] for _ in range(3))
    v = [make(n).abs_() for n in sizes]
    w = [make(n, torch.bfloat16) for n in sizes]
    for ts in (gr, v, m):
        for t in ts[:1]:
            t[0] = 0.0  # an element that has never had a gradient only decays
    old = [[t.double().clone() for t in ts] for ts in (p, m, v, gr)]
    lr, b1, b2, eps, wd, t = 1e-2, 0.9, 0.95, 1e-8, 0.1, 3
    c1, c2 = 1 - b1**t, 1 - b2**t
    adamw_update(p, m, v, gr, w, lr=lr, b1=b1, b2=b2, eps=eps, weight_decay=wd, c1=c1, c2=c2)
    u = 2.0**-24
    for i in range(len(sizes)):
        p0, m0, v0, g0 = (ts[i] for ts in old)
        m1, v1 = b1 * m0 + (1 - b1) * g0, b2 * v0 + (1 - b2) * g0 * g0
        step = lr / c1 * m1 / ((v1 / c2).sqrt() + eps)
        p1 = p0 * (1 - lr * wd) - step
        # a rounding for each coefficient, product and sum; the step adds those of the root, the sum and the quotients
        dm, dv = 4 * u * ((b1 * m0).abs() + ((1 - b1) * g0).abs()), 5 * u * v1
        assert bool(((m[i].double() - m1).abs() <= dm).all()) and bool(((v[i].double() - v1).abs() <= dv).all())
        dstep = 12 * u * step.abs() + lr / c1 * dm / ((v1 / c2).sqrt() + eps)
        assert bool(((p[i].double() - p1).abs() <= 4 * u * (p0.abs() + step.abs()) + dstep).all())
        assert torch.equal(w[i], p[i].to(torch.bfloat16))


def test_adamw_refuses_lists_that_do_not_match():
    t = [torch.zeros(4)]
    with pytest.raises(ValueError):
        adamw_update(t, t, t, t, t + t, lr=1e-2, b1=0.9, b2=0.95, eps=1e-8, weight_decay=0.0, c1=0.1, c2=0.05)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [8, 2040, 148 * 8 * 2048 - 8, 148 * 16 * 2048 + 8, 148 * 40 * 2048 + 2056])
def test_sgd_update_at_the_edges_of_its_grid(n):
    from moonep_b200.ops.moe_ops import sgd_update

    g = torch.Generator(device="cuda").manual_seed(n)
    w0 = torch.randn(n, generator=g, device="cuda").to(torch.bfloat16)
    gr = torch.randn(n, generator=g, device="cuda")
    w = torch.cat([w0, w0[:8]])
    sgd_update(w[:n], gr, 0.25)
    # the product is exact, the difference rounded to fp32 (2^-24) and to bf16, whose 8-bit mantissa gives 2^-8
    want = w0.double() - 0.25 * gr.double()
    assert bool(((w[:n].double() - want).abs() <= (2.0**-8 + 2.0**-23) * want.abs()).all())
    assert torch.equal(w[n:], w0[:8])  # nothing past the end
