"""Dense helpers of the MoE layer and block: batched expert transposes, the SwiGLU backward, weight updates, the router.

CUDA tensors run the kernels of ``csrc/moe_kernels.cu`` and ``csrc/router.cu``; CPU tensors run the same arithmetic in torch.
"""

from __future__ import annotations

import ctypes

import torch

from . import _lib


def transpose_experts(src: torch.Tensor, dst: torch.Tensor, col0: int = 0, active=None) -> torch.Tensor:
    """``dst[n, j, col0 + i] = src[n, i, j]``; ``src`` is ``[n, d0, d1]`` bf16, ``dst`` ``[n, d1, >= col0 + d0]``.
    ``active`` (int32 ``[n]``, optional): matrices whose entry is negative are skipped."""
    n, d0, d1 = (int(v) for v in src.shape)
    assert dst.shape[0] == n and dst.shape[1] == d1 and dst.shape[2] >= col0 + d0 and dst.is_contiguous()
    if active is not None:
        assert active.dtype == torch.int32 and active.numel() == n and active.is_contiguous()
    if not src.is_cuda:
        for i in range(n):
            if active is None or int(active[i]) >= 0:
                dst[i, :, col0 : col0 + d0] = src[i].transpose(0, 1)
        return dst
    assert src.is_contiguous() and src.dtype == torch.bfloat16 and dst.dtype == torch.bfloat16
    with _lib.on_device(src.device):
        rc = _lib.load().moonep_transpose_experts(
            src.data_ptr(), dst.data_ptr(), n, d0, d1, int(dst.shape[2]), int(dst.shape[1]) * int(dst.shape[2]), int(col0),
            None if active is None else active.data_ptr(), _lib.current_stream(),
        )  # fmt: skip
    _lib.check(rc, "moonep_transpose_experts")
    return dst


def swiglu_bwd(a, u, g, w, total_rows, dadu, hsw, dgate) -> None:
    """See ``csrc/moe_kernels.cu``: fills ``dadu[rows, 2I]``, ``hsw[rows, I]``, ``dgate[rows]`` for rows < total."""
    rows, I = (int(v) for v in a.shape)
    if not a.is_cuda:
        n = int(total_rows[0]) if total_rows is not None else rows
        af, uf, gf = a[:n].float(), u[:n].float(), g[:n].float()
        s = torch.sigmoid(af)
        h = af * s * uf
        dgate[:n] = (gf * h).sum(dim=1)
        dh = gf * w[:n, None]
        dadu[:n, :I] = (dh * uf * s * (1 + af * (1 - s))).to(dadu.dtype)
        dadu[:n, I:] = (dh * af * s).to(dadu.dtype)
        hsw[:n] = (h * w[:n, None]).to(hsw.dtype)
        return
    for t in (a, u, g, dadu, hsw):
        assert t.is_contiguous() and t.dtype == torch.bfloat16
    assert w.dtype == torch.float32 and dgate.dtype == torch.float32 and w.is_contiguous() and dgate.is_contiguous()
    with _lib.on_device(a.device):
        rc = _lib.caller("moonep_swiglu_bwd")(
            a.data_ptr(), u.data_ptr(), g.data_ptr(), w.data_ptr(), 0 if total_rows is None else total_rows.data_ptr(),
            rows, I, dadu.data_ptr(), hsw.data_ptr(), dgate.data_ptr(), _lib.current_stream(),
        )  # fmt: skip
    _lib.check(rc, "moonep_swiglu_bwd")


_UPDATE_TENSORS = 3  # weights per launch of the update kernels


def sgd_update(w: torch.Tensor, g: torch.Tensor, lr: float) -> None:
    """``w -= lr * g`` for a bf16 weight tensor and its fp32 gradient (same shape, contiguous)."""
    sgd_updates([w], [g], lr)


def sgd_updates(weights, grads, lr: float) -> None:
    """``w -= lr * g`` for any number of bf16 weights and their fp32 gradients, the kernel's share in one launch."""
    todo = []
    for w, g in zip(weights, grads):
        assert w.shape == g.shape
        if not w.is_cuda or w.numel() % 8 != 0 or (w.data_ptr() | g.data_ptr()) % 16 != 0:
            w.add_(g, alpha=-lr)
            continue
        assert w.is_contiguous() and g.is_contiguous() and w.dtype == torch.bfloat16 and g.dtype == torch.float32
        todo.append((w, g))
    while todo:
        some = [t for t in todo if t[0].device == todo[0][0].device][:_UPDATE_TENSORS]
        todo = [t for t in todo if all(t is not s for s in some)]
        n = len(some)
        ws, gs = ((ctypes.c_void_p * n)(*[t[i].data_ptr() for t in some]) for i in (0, 1))
        sizes = (ctypes.c_longlong * n)(*[w.numel() for w, _ in some])
        with _lib.on_device(some[0][0].device):
            rc = _lib.load().moonep_sgd_update(n, ws, gs, sizes, float(lr), _lib.current_stream())
        _lib.check(rc, "moonep_sgd_update")


def adamw_update(masters, exp_avgs, exp_avg_sqs, grads, weights, *, lr, b1, b2, eps, weight_decay, c1, c2) -> None:
    """One AdamW step of any number of weights: fp32 ``masters`` and moments are updated from the fp32 ``grads`` and the
    rounded masters stored to the bf16 ``weights``.  ``c1``, ``c2``: bias corrections ``1 - b**t``."""
    tensors = [list(ts) for ts in (masters, exp_avgs, exp_avg_sqs, grads, weights)]
    if len({len(ts) for ts in tensors}) != 1:
        raise ValueError(f"adamw_update: lists of {[len(ts) for ts in tensors]} tensors")
    for i in range(0, len(tensors[4]), _UPDATE_TENSORS):
        _adamw_step([ts[i : i + _UPDATE_TENSORS] for ts in tensors], lr, b1, b2, eps, weight_decay, c1, c2)


def _adamw_step(tensors, lr, b1, b2, eps, weight_decay, c1, c2) -> None:
    weights = tensors[4]
    kernel = all(
        t.is_cuda and t.is_contiguous() and t.numel() == w.numel() and t.device == weights[0].device
        and t.dtype == (torch.bfloat16 if ts is weights else torch.float32)
        and t.numel() % 4 == 0 and t.data_ptr() % (8 if ts is weights else 16) == 0
        for ts in tensors for t, w in zip(ts, weights)
    )  # fmt: skip
    if not kernel:
        for p, m, v, g, w in zip(*tensors):
            if weight_decay:
                p.mul_(1.0 - lr * weight_decay)
            m.mul_(b1).add_(g, alpha=1.0 - b1)
            v.mul_(b2).addcmul_(g, g, value=1.0 - b2)
            p.addcdiv_(m, (v / c2).sqrt_().add_(eps), value=-lr / c1)
            w.copy_(p)
        return
    n = len(weights)
    ptrs = [(ctypes.c_void_p * n)(*[t.data_ptr() for t in ts]) for ts in tensors]
    sizes = (ctypes.c_longlong * n)(*[t.numel() for t in weights])
    with _lib.on_device(weights[0].device):
        rc = _lib.load().moonep_adamw_update(n, *ptrs, sizes, lr / c1, b1, b2, eps, 1.0 - lr * weight_decay, c2,
                                             _lib.current_stream())  # fmt: skip
    _lib.check(rc, "moonep_adamw_update")


ROUTER_MAX_EXPERTS, ROUTER_MAX_TOPK = 64, 32  # of the router kernels


def router_kernel_supports(x: torch.Tensor, weight: torch.Tensor, k: int) -> bool:
    """Whether ``csrc/router.cu`` can take this call."""
    return (
        x.is_cuda and weight.is_cuda and x.device == weight.device and x.dim() == 2 and weight.dim() == 2
        and x.dtype == torch.bfloat16 and weight.dtype == torch.float32 and x.is_contiguous() and weight.is_contiguous()
        and x.shape[0] >= 1 and x.shape[1] == weight.shape[1] and x.shape[1] >= 8 and x.shape[1] % 8 == 0
        and 1 <= k <= min(int(weight.shape[0]), ROUTER_MAX_TOPK) and weight.shape[0] <= ROUTER_MAX_EXPERTS
        and x.data_ptr() % 16 == 0 and weight.data_ptr() % 16 == 0
    )  # fmt: skip


def router_kernel_pays(tokens: int, hidden: int, num_experts: int, k: int) -> bool:
    """Whether the router kernels are the faster ones, forward and with the backward pass.

    Their two launches replace thirty, but a CTA reads the whole weight for its eight tokens, and every selection of a token reads
    a row of it in the backward pass, where the operations have tiled matrix products.  Device time, kernels and operations, us
    (of 2551 sizes: S 1 to 16384, H 256 to 16384, 4 to 64 experts, 1 to 32 selections):

    * size of the weight, forward pass: S=1 H=7168, 16 experts 47 and 58, 24 experts 68 and 54, 64 experts 164 and 58;
      S=64 H=7168, 32 experts 86 and 101, 48 experts 125 and 107, 64 experts 162 and 107
    * forward and backward pass: S=16384 H=7168 K=8, 32 experts 1192 and 1292, 48 experts 1589 and 1532, 64 experts 2007 and 1591
    * selections, forward and backward pass: S=16384 H=7168, 32 experts, K=12 1.02 of the operations' time, K=16 1.31, K=32 2.7;
      S=16384 H=2048, 64 experts, K=16 1.14
    """
    return k <= 12 and num_experts * hidden <= (16 if tokens < 64 else 32) * 7168


def router_forward(x: torch.Tensor, weight: torch.Tensor, k: int, keep_gates: bool = False, keep_x: bool = False):
    """``(gates [S, k] fp32, topk [S, k] int32, tokens_per_expert [E] int32)`` of logits ``x @ weight.T``, then copies of
    ``gates`` and ``topk`` and a copy of ``x``, each None unless asked for."""
    (S, H), E = x.shape, int(weight.shape[0])
    gates = torch.empty(S, k, dtype=torch.float32, device=x.device)
    topk = torch.empty(S, k, dtype=torch.int32, device=x.device)
    tpe = torch.empty(E, dtype=torch.int32, device=x.device)
    gates_kept, topk_kept = (torch.empty_like(gates), torch.empty_like(topk)) if keep_gates else (None, None)
    x_kept = torch.empty_like(x) if keep_x else None
    with _lib.on_device(x.device):
        rc = _lib.load().moonep_router_fwd(
            x.data_ptr(), weight.data_ptr(), S, H, E, k, gates.data_ptr(), topk.data_ptr(), tpe.data_ptr(),
            x_kept.data_ptr() if keep_x else None, gates_kept.data_ptr() if keep_gates else None,
            topk_kept.data_ptr() if keep_gates else None, _lib.current_stream(),
        )  # fmt: skip
    _lib.check(rc, "moonep_router_fwd")
    return gates, topk, tpe, gates_kept, topk_kept, x_kept


def router_backward(x, weight, gates, topk, dgates, num_experts: int, want_dx: bool, want_dw: bool):
    """Gradients of ``router_forward``'s gates: ``(dx [S, H] bf16 or None, dweight [E, H] fp32 or None)``.  ``weight`` is only
    read for the first and ``x`` for the second; without them they may be None."""
    (S, k), H = gates.shape, (x if want_dw else weight).shape[1]
    dx = torch.empty(S, H, dtype=torch.bfloat16, device=gates.device) if want_dx else None
    dw = torch.empty(num_experts, H, dtype=torch.float32, device=gates.device) if want_dw else None
    with _lib.on_device(gates.device):
        rc = _lib.load().moonep_router_bwd(
            x.data_ptr() if want_dw else None, weight.data_ptr() if want_dx else None, gates.data_ptr(), topk.data_ptr(),
            dgates.data_ptr(), S, H, num_experts, k, dx.data_ptr() if want_dx else None, dw.data_ptr() if want_dw else None,
            _lib.current_stream(),
        )  # fmt: skip
    _lib.check(rc, "moonep_router_bwd")
    return dx, dw
