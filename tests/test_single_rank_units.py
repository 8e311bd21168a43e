"""One rank's dispatch moves several short rows through a stage at a time: as many as fit, make equal shares, and are left."""

import pytest
import torch

from moonep_b200 import Buffer


@pytest.mark.gpu
@pytest.mark.parametrize("S,H,K,E,pad", [
    (1, 8, 3, 4, 8), (148 * 6 + 1, 256, 2, 5, 8), (148 * 48, 512, 3, 6, 4), (148 * 48 + 3, 504, 3, 6, 4), (9000, 1024, 2, 9, 16),
    (3000, 2048, 4, 8, 16), (701, 4104, 2, 7, 8), (3000, 4096, 2, 7, 8), (300, 8192, 2, 7, 8), (200, 8200, 2, 7, 8),
    (5000, 40, 32, 40, 2),
])  # fmt: skip
def test_every_row_arrives(S, H, K, E, pad):
    buf = Buffer(S, H, K, E, 1, token_padding=pad)
    g = torch.Generator(device="cuda").manual_seed(S + H)
    topk = torch.rand(S, E, generator=g, device="cuda").topk(K, dim=1).indices.int()
    tpe = torch.bincount(topk.flatten().long(), minlength=E).int()
    gates = torch.rand(S, K, generator=g, device="cuda")
    plan = None
    for turn in range(4):  # fresh, staged, replayed, fresh
        x = torch.randn(S, H, generator=g, device="cuda").to(torch.bfloat16)
        buf._require_ctx()["hidden_buf_local"].fill_(7.0)
        if turn == 2:
            rows, w, _, _ = buf.dispatch(x, gates, plan=plan, zero_copy=True)
        else:
            rows, w, cu, plan = buf.dispatch(x, gates, topk, tpe, zero_copy=turn != 1)
        buf.check_status()
        at = torch.where(plan.dst < 0, -plan.dst - 1, plan.dst).long()
        assert torch.equal(rows[at], x.repeat_interleave(K, 0)) and torch.equal(w[at], gates.flatten())
        pads = torch.ones(int(cu[-1]), dtype=torch.bool, device="cuda")
        pads[at] = False
        assert not bool(rows[: int(cu[-1])][pads].any())
        ctx = buf._require_ctx()
        flags = ctx["meta_buf"][ctx["ROWFLAG_OFF"] : ctx["ROWFLAG_OFF"] + int(cu[-1])]
        assert bool((flags == flags[0]).all()) and int(flags[0]) == turn + 1
    buf.destroy()
