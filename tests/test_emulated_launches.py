"""Emulated ranks merge the roles that need nothing of a peer into one launch (OWN with SEND, FOLD with PUSH).
``MOONEP_PHASED=1`` launches every role by itself: both have to give the same rows, flags, plans and sums, bit for bit."""

import pytest
import torch

from moonep_b200 import Buffer
from moonep_b200.models.routing import make_routing
from moonep_b200.parallel.world import LocalWorld

# S, H, K, experts per rank, B, num_sms, padding; rows: 16-byte words, several pieces per row, not 16-byte multiples
SHAPES = [(5, 8, 1, 2, 1, 2, 8), (301, 264, 4, 4, 2, 1, 16), (33, 9224, 5, 3, 2, 3, 8), (200, 1544, 32, 2, 1, 140, 16),
          (64, 1002, 3, 4, 2, 4, 4), (700, 520, 6, 8, 4, 8, 32)]  # fmt: skip


def _passes(R, S, H, K, epn, B, num_sms, pad):
    E, world = R * epn, LocalWorld(R, "cuda")

    def body(r):
        buf = Buffer(S, H, K, E, R, num_sms=num_sms, token_padding=pad, B=B, world=world.view(r))
        ctx, got = buf._require_ctx(), []
        topk, tpe, gates = make_routing("duplicate_topk" if K > E else "biased", S, K, E, R, r, bias=1.0, seed=3, device="cuda")
        g = torch.Generator(device="cuda").manual_seed(r)
        ctx["hidden_buf_local"].fill_(7.0)
        plan = None
        for turn in range(3):  # fresh, replayed, fresh
            x = torch.randn(S, H, generator=g, device="cuda").to(torch.bfloat16)
            if turn == 1:
                rows, w, _, _ = buf.dispatch(x, gates, plan=plan, zero_copy=True)
            else:
                rows, w, cu, plan = buf.dispatch(x, gates, topk, tpe, zero_copy=True)
            base = r * ctx["meta_chunk_padded"] + ctx["ROWFLAG_OFF"]
            flags = ctx["meta_buf"][base : base + int(cu[-1])]
            y = (rows.float() * (torch.arange(rows.shape[0], device="cuda") % 7 + 0.3)[:, None]).to(torch.bfloat16)
            out, back, _ = buf.combine(plan, y, w)
            buf.synchronize()
            world.view(r).step()
            order = plan.dup_groups[: int(plan.dup_counts[0]), 0].sort().values
            got += [t.clone() for t in (rows, w, cu, plan.dst, order, flags, out, back)]
        buf.destroy()
        return got

    return world.run(body)


@pytest.mark.gpu
@pytest.mark.parametrize("R", [2, 4])
@pytest.mark.parametrize("shape", SHAPES, ids=str)
def test_merged_launches_give_what_single_roles_give(shape, R, monkeypatch):
    merged = _passes(R, *shape)
    monkeypatch.setenv("MOONEP_LOCAL_SMS", "5")  # fewer SMs than there are senders for some
    few = _passes(R, *shape)
    monkeypatch.delenv("MOONEP_LOCAL_SMS")
    monkeypatch.setenv("MOONEP_PHASED", "1")
    single = _passes(R, *shape)
    for r in range(R):
        for name, a, b, c in zip(("rows", "weights", "cu", "dst", "groups", "flags", "out", "gates") * 3, merged[r], few[r], single[r]):
            assert torch.equal(a, c) and torch.equal(b, c), f"rank {r}: {name}"
