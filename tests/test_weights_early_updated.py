"""Products that ask for their weights before the kernel ahead of them has ended, where the weights were changed by the kernel ahead
of that one: they have to be the new ones.  Behind the SwiGLU product, a replayed dispatch and the weight gradients, as in a layer."""

import pytest
import torch

from moonep_b200 import Buffer
from moonep_b200.ops.grouped_gemm import WGRAD_STORE, grouped_gemm, grouped_gemm_kn, grouped_wgrad_rows

TURNS = 6


def _passes(update, ahead, product):
    """The product of every turn, with early and with late weights; everything is queued before the first kernel runs."""
    got = []
    for early in (True, False):
        torch.cuda.synchronize()
        torch.cuda._sleep(20_000_000)
        outs = []
        for turn in range(TURNS):
            update(turn)
            ahead()
            outs.append(product(early))
        got.append(outs)
    return got


def _check(got):
    early, late = got
    assert all(torch.equal(a, b) for a, b in zip(early, late))
    assert not any(torch.equal(a, b) for a, b in zip(late, late[1:]))  # stale weights would show


def _randn(g, *shape, scale=1.0):
    return (torch.randn(*shape, generator=g, device="cuda") * scale).bfloat16()


@pytest.mark.gpu
@pytest.mark.parametrize("E,rows,H,I", [(16, 128, 2048, 1024), (8, 256, 4096, 512), (3, 128, 512, 256)])
def test_down_projection_behind_the_swiglu_product(E, rows, H, I):
    g = torch.Generator(device="cuda").manual_seed(E)
    cu = (torch.arange(1, E + 1, device="cuda") * rows).int()
    x, gate, up = _randn(g, E * rows, H), _randn(g, E, I, H, scale=H**-0.5), _randn(g, E, I, H, scale=H**-0.5)
    downs, down = [_randn(g, E, H, I, scale=I**-0.5) for _ in range(2)], torch.empty(E, H, I, device="cuda").bfloat16()
    scale, h = torch.rand(E * rows, generator=g, device="cuda"), torch.empty(E * rows, I, device="cuda").bfloat16()
    _check(_passes(lambda turn: down.copy_(downs[turn % 2]),
                   lambda: grouped_gemm(x, gate, cu, w_up=up, mode="swiglu", out=h, pair=False),
                   lambda early: grouped_gemm(h, down, cu, mode="scale", row_scale=scale, pair=False, weights_early=early)))  # fmt: skip


@pytest.mark.gpu
@pytest.mark.parametrize("S,H,K,E,I", [(256, 2048, 4, 16, 1024), (64, 1024, 2, 4, 512), (1000, 4096, 2, 2, 512)])
@pytest.mark.parametrize("behind", ["dispatch", "wgrad"])
def test_activation_gradients_behind_what_runs_ahead_of_them(behind, S, H, K, E, I):
    g = torch.Generator(device="cuda").manual_seed(S)
    buf = Buffer(S, H, K, E, 1, num_sms=8, token_padding=128)
    topk = torch.rand(S, E, generator=g, device="cuda").topk(K).indices.int()
    tpe = torch.bincount(topk.flatten(), minlength=E).int()
    x, gates = _randn(g, S, H), torch.rand(S, K, generator=g, device="cuda")
    rows, _, cu, plan = buf.dispatch(x, gates, topk, tpe, zero_copy=True)
    n, G = int(cu[-1]), int(cu.numel())
    ws, w = [_randn(g, G, H, I, scale=H**-0.5) for _ in range(2)], torch.empty(G, H, I, device="cuda").bfloat16()
    right = _randn(g, rows.shape[0], I)
    grads = torch.empty(G, H, I, device="cuda")
    ptrs = torch.tensor([t.data_ptr() for t in grads], device="cuda")
    flags = torch.full((G,), WGRAD_STORE, dtype=torch.int32, device="cuda")
    if behind == "dispatch":
        ahead = lambda: buf.dispatch(x, None, plan=plan, zero_copy=True)  # noqa: E731
    else:
        ahead = lambda: grouped_wgrad_rows(rows, right, cu, ptrs, flags)  # noqa: E731
    _check(_passes(lambda turn: w.copy_(ws[turn % 2]), ahead,
                   lambda early: grouped_gemm_kn(rows, [w], cu, pair=False, weights_early=early)[:n]))  # fmt: skip
    buf.check_status()
    buf.destroy()
