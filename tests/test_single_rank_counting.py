"""One rank's dispatch: every CTA counts the routing entries before its tokens, some of them asked for before it knows the group
layout.  Rows come in routing order with few and many entries, skewed ones, entries left over and unaligned ones."""

import pytest
import torch

from moonep_b200 import Buffer


@pytest.mark.gpu
@pytest.mark.parametrize("S,H,K,E,pad,skew", [
    (4097, 16, 1, 1, 1, 0.0), (1400, 8, 3, 5, 8, 0.0), (40001, 8, 3, 7, 16, 0.97), (32768, 8, 8, 9, 1, 1.0),
    (9001, 24, 5, 64, 4, 0.5), (4099, 40, 8, 257, 128, 0.0), (3001, 7168, 8, 130, 16, 0.0),
    (5000, 8, 4, 1500, 2, 0.2), (5003, 12, 3, 31, 1, 0.3),  # many experts, rows that are not 16-byte multiples
])  # fmt: skip
def test_rows_follow_the_routing_order(S, H, K, E, pad, skew):
    buf = Buffer(S, H, K, E, 1, token_padding=pad)
    g = torch.Generator(device="cuda").manual_seed(S + E)
    topk = torch.randint(0, E, (S, K), generator=g, device="cuda", dtype=torch.int32)
    topk[torch.rand(S, K, generator=g, device="cuda") < skew] = E - 1
    tpe = torch.bincount(topk.flatten().long(), minlength=E).int()
    x = torch.randn(S, H, generator=g, device="cuda").to(torch.bfloat16)
    flat, ends = topk.flatten().long(), ((tpe.long() + pad - 1) // pad * pad).cumsum(0)
    start = ends - (tpe.long() + pad - 1) // pad * pad
    order = torch.argsort(flat, stable=True)
    want = torch.empty(S * K, dtype=torch.long, device="cuda")
    want[order] = torch.arange(S * K, device="cuda") - (tpe.long().cumsum(0) - tpe)[flat[order]] + start[flat[order]]
    for shift in (0, 1):  # aligned, and not readable 16 bytes at a time
        entries = torch.empty(S * K + 4, dtype=torch.int32, device="cuda")[shift : shift + S * K].view(S, K).copy_(topk)
        rows, _, cu, plan = buf.dispatch(x, None, entries, tpe, zero_copy=True)
        buf.check_status()
        assert torch.equal(torch.where(plan.dst < 0, -plan.dst - 1, plan.dst).long(), want) and torch.equal(cu[:E].long(), ends)
        assert torch.equal(rows[want], x.repeat_interleave(K, 0))
        rows.fill_(3.0)
        rows, _, _, _ = buf.dispatch(-x, None, plan=plan, zero_copy=True)
        assert torch.equal(rows[want], -x.repeat_interleave(K, 0))
    buf.destroy()
