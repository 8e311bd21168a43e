"""Dispatch and combine kernels of a single rank (csrc/single_rank.cu) at the edges of their tiling, against the host
planner and the two-rounding model: pieces of rows, tokens per CTA, steps of 384 entries, 512 groups scanned at a time, rows
and routing that are not 16-byte aligned, tokens handed out between CTAs, replayed plans, token counts that do not match the
routing, sizes that take the general kernels."""

import pytest
import torch

from moonep_b200 import Buffer
from moonep_b200.constants import FLAG_SENT
from moonep_b200.errors import MoonEPIndexError, MoonEPTimeoutError
from tests.harness import Case, assert_within_ulp, check_dispatch_records, expected_combine, run_round_trip

pytestmark = pytest.mark.gpu

CASES = [
    Case("one_token_many_pads", S=1, K=1, epn=3, H=8, token_padding=128, routing="single_expert"),
    Case("fewer_tokens_than_ctas", S=147, K=3, epn=5, H=264, token_padding=16, routing="biased"),
    Case("one_cta_with_one_token", S=149, K=2, epn=8, H=4104, token_padding=1, routing="softmax"),
    Case("two_pieces_per_row", S=40, K=4, epn=6, H=8200, token_padding=32, routing="zipf"),
    Case("three_pieces_per_row", S=40, K=4, epn=6, H=16392, token_padding=32, routing="zipf"),
    Case("several_steps_per_cta", S=12000, K=8, epn=16, H=64, token_padding=64, routing="zipf"),
    Case("twelve_tokens_per_step", S=300, K=32, epn=40, H=32, token_padding=8, routing="softmax"),
    Case("one_entry_past_a_step", S=149 * 129, K=3, epn=8, H=16, token_padding=4, routing="softmax"),  # 130 tokens per CTA
    Case("one_scan_of_groups", S=700, K=2, epn=512, H=16, token_padding=4, routing="softmax", B=1),
    Case("three_scans_of_groups", S=700, K=2, epn=1100, H=16, token_padding=4, routing="softmax", B=1),
    Case("rows_of_40_bytes", S=333, K=5, epn=7, H=20, token_padding=16, routing="biased"),
    Case("odd_rows", S=50, K=2, epn=4, H=13, token_padding=4, routing="softmax"),
]


@pytest.mark.parametrize("zero_copy", [False, True])
@pytest.mark.parametrize("case", CASES, ids=lambda c: c.name)
def test_single_rank_round_trip(case, zero_copy):
    recs = run_round_trip(case, 1, "cuda", zero_copy=zero_copy,
                          expert_scale=lambda rec, r, E: (torch.arange(rec["hidden_nvsh"].shape[0]) % 5 + 1).float())  # fmt: skip
    _, dst_pos, _, _ = check_dispatch_records(case, 1, recs)
    scale = [(torch.arange(recs[0]["layout"]["NvS"]) % 5 + 1).float()]
    want = expected_combine(case, 1, recs, dst_pos, scale)
    assert_within_ulp(recs[0]["out"], want[0], max_ulps=1, what="combine")
    assert torch.equal(recs[0]["weights_back"], recs[0]["w"])


def _inputs(S, H, K, E, shift):
    """Routing and rows that start ``shift`` elements into their storage (contiguous, not 16-byte aligned)."""
    g = torch.Generator(device="cuda").manual_seed(3)
    topk = torch.rand(S, E, generator=g, device="cuda").topk(K, dim=1).indices.to(torch.int32)
    topk = torch.empty(S * K + shift, dtype=torch.int32, device="cuda")[shift:].view(S, K).copy_(topk)
    x = torch.empty(S * H + shift, dtype=torch.bfloat16, device="cuda")[shift:].view(S, H)
    x.copy_(torch.randn(S, H, generator=g, device="cuda"))
    return x, topk, torch.bincount(topk.flatten().long(), minlength=E).to(torch.int32)


@pytest.mark.parametrize("shift", [0, 1, 4])
@pytest.mark.parametrize("S,H,K,E,pad", [(1, 64, 2, 4, 8), (500, 520, 3, 9, 16), (3000, 64, 6, 12, 1),
                                         # several pieces per row, in words of 16 (or 2, read), 8, 4 and 2 bytes
                                         (20, 2056, 3, 5, 8), (150, 1028, 2, 4, 8), (33, 1002, 2, 4, 4), (9, 515, 4, 5, 2)])  # fmt: skip
def test_replay_and_unaligned_inputs(S, H, K, E, pad, shift):
    buf = Buffer(S, H, K, E, 1, token_padding=pad)
    x, topk, tpe = _inputs(S, H, K, E, shift)
    gates = torch.rand(S, K, device="cuda")
    ctx = buf._require_ctx()
    ctx["hidden_buf_local"].fill_(7.0)
    ctx["weights_buf_local"].fill_(3)
    rows, w, cu, plan = buf.dispatch(x, gates, topk, tpe)
    # a staged dispatch returns the whole shard and its weights, rows that no group uses included
    assert torch.equal(rows, ctx["hidden_buf_local"]) and torch.equal(w.view(torch.int32), ctx["weights_buf_local"])
    assert bool((rows[int(cu[-1]) :] == 7.0).all())
    x2 = torch.empty_like(x).copy_(-x)
    buf._require_ctx()["hidden_buf_local"].fill_(7.0)
    rows2, w2, _, _ = buf.dispatch(x2, gates, plan=plan, zero_copy=True)
    loff = torch.where(plan.dst < 0, -plan.dst - 1, plan.dst).long()
    end = int(cu[-1])
    assert torch.equal(rows[loff], x.repeat_interleave(K, 0)) and torch.equal(rows2[loff], x2.repeat_interleave(K, 0))
    pads = torch.ones(end, dtype=torch.bool, device="cuda")
    pads[loff] = False
    assert not bool(rows2[:end][pads].any()) and torch.equal(w2[loff], gates.flatten())
    y = torch.randn(buf._require_ctx()["NvS"], H, device="cuda").to(torch.bfloat16)
    out, back, _ = buf.combine(plan, y, w2.clone())
    want = torch.zeros(S, H, device="cuda")
    for k in range(K):  # the kernel's order: fp32, ascending k, rounded once
        want += y[loff.view(S, K)[:, k]].float()
    assert torch.equal(out, want.to(torch.bfloat16)) and torch.equal(back, gates)
    buf.synchronize()
    buf.destroy()


@pytest.mark.parametrize("ctas", ["1", "2", "3", None])
@pytest.mark.parametrize("var", ["MOONEP_NUM_SMS_DEDUP", "MOONEP_LOCAL_SMS"])
@pytest.mark.parametrize("S,H,K,E,pad,shift,hot", [
    (2000, 2056, 2, 9, 4, 0, True),   # more units of a copy warp than it remembers, and tokens to hand out on every grid
    (250, 16392, 3, 8, 8, 0, False),  # the same with rows of three pieces
    (100, 2056, 2, 100, 128, 0, False),  # more grabs of pad rows than a warp remembers
    (1500, 1032, 2, 9, 16, 1, True),  # without bulk copies
])  # fmt: skip
def test_tokens_and_pads_handed_out_between_ctas(S, H, K, E, pad, shift, hot, var, ctas, monkeypatch):
    """Fresh, staged and replayed dispatches in a row on one Buffer: every row, pad row and row flag, on grids of one to
    three CTAs and of every SM."""
    if ctas is None and var == "MOONEP_LOCAL_SMS":
        pytest.skip("the same as the other switch unset")
    if ctas is not None:
        monkeypatch.setenv(var, ctas)
    buf = Buffer(S, H, K, E, 1, token_padding=pad)
    ctx = buf._require_ctx()
    be = ctx["_backend"]
    g = torch.Generator(device="cuda").manual_seed(S)
    flags = ctx["meta_buf"][ctx["ROWFLAG_OFF"] :][: ctx["NvS"]]
    plan = None
    for turn in range(6):
        fresh, staged = turn % 3 != 2, turn % 3 == 1
        if fresh:
            lg = torch.rand(S, E, generator=g, device="cuda") * (torch.arange(E, device="cuda") < 4 + turn if hot else 1)
            topk = lg.topk(K, dim=1).indices.to(torch.int32)
            tpe = torch.bincount(topk.flatten().long(), minlength=E).to(torch.int32)
        x = torch.empty(S * H + shift, dtype=torch.bfloat16, device="cuda")[shift:].view(S, H)
        x.copy_(torch.randn(S, H, generator=g, device="cuda"))
        gates = torch.rand(S, K, generator=g, device="cuda")
        ctx["hidden_buf_local"].fill_(7.0)
        if fresh:
            rows, w, cu, plan = buf.dispatch(x, gates, topk, tpe, zero_copy=not staged)
        else:
            rows, w, _, _ = buf.dispatch(x, gates, plan=plan, zero_copy=True)
        end = int(cu[-1])
        loff = torch.where(plan.dst < 0, -plan.dst - 1, plan.dst).long()
        assert torch.equal(rows[loff], x.repeat_interleave(K, 0)) and torch.equal(w[loff], gates.flatten())
        assert int(torch.unique(loff).numel()) == S * K and torch.equal(plan.src_info[loff].long(), torch.arange(S * K, device="cuda"))
        pads = torch.ones(end, dtype=torch.bool, device="cuda")
        pads[loff] = False
        assert not bool(rows[:end][pads].any()) and not bool(w[:end][pads].any()) and bool((rows[end:] == 7.0).all())
        assert bool((flags[:end] == be.epoch[FLAG_SENT]).all())
        out, back, _ = buf.combine(plan, rows, w)
        want = torch.zeros(S, H, device="cuda")
        for _ in range(K):
            want += x.float()
        assert torch.equal(out, want.to(torch.bfloat16)) and torch.equal(back, gates)
        buf.synchronize()
    buf.destroy()


@pytest.mark.parametrize("S,K,E,single", [(32768, 8, 16, True), (32769, 8, 16, False), (64, 1, 4096, True), (64, 1, 4097, False)])
def test_on_each_side_of_the_single_rank_limits(S, K, E, single):
    """262144 routing entries and 4096 experts are the most the single-rank dispatch takes; beyond, the general kernels
    make the same plan, which the single-rank combine reads."""
    H = 8
    buf = Buffer(S, H, K, E, 1, token_padding=2, B=1)
    be = buf._require_ctx()["_backend"]
    x, topk, tpe = _inputs(S, H, K, E, 0)
    gates = torch.rand(S, K, device="cuda")
    be.profile(True)
    rows, w, cu, plan = buf.dispatch(x, gates, topk, tpe)
    loff = torch.where(plan.dst < 0, -plan.dst - 1, plan.dst).long()
    rows2, w2, _, _ = buf.dispatch(-x, gates, plan=plan, zero_copy=True)
    out, back, _ = buf.combine(plan, rows2, w2, zero_copy=True)
    tags = set(be.phase_times())
    assert ("dispatch_single" in tags) == single and ("dispatch_fused" in tags) != single and "combine_single" in tags
    # rows of an expert in the order of the routing entries
    flat = topk.flatten().long()
    padded = (tpe.long() + 1) // 2 * 2
    first = padded.cumsum(0) - padded
    order = torch.sort(flat, stable=True).indices
    want = torch.empty(S * K, dtype=torch.long, device="cuda")
    want[order] = torch.arange(S * K, device="cuda") - (tpe.long().cumsum(0) - tpe)[flat[order]] + first[flat[order]]
    assert torch.equal(loff, want) and int(cu[-1]) == int(padded.sum())
    assert torch.equal(rows[loff], x.repeat_interleave(K, 0)) and torch.equal(w[loff], gates.flatten())
    assert torch.equal(rows2[loff], -x.repeat_interleave(K, 0))
    acc = torch.zeros(S, H, device="cuda")
    for _ in range(K):
        acc -= x.float()
    assert torch.equal(out, acc.to(torch.bfloat16)) and torch.equal(back, gates)
    buf.synchronize()
    buf.destroy()


@pytest.mark.parametrize("K", [1, 3, 6])
def test_combine_takes_rows_as_their_blocks_are_finished(K):
    """``combine(ready=...)`` on one rank: behind a product that counts its row blocks, and behind one that never finishes
    the last count, which is a timeout after which the Buffer works again."""
    from moonep_b200.ops.grouped_gemm import grouped_gemm

    S, H, E = 300, 256, 8
    buf = Buffer(S, H, K, E, 1, token_padding=128, B=1)
    be = buf._require_ctx()["_backend"]
    x, topk, tpe = _inputs(S, H, K, E, 0)
    rows, _, cu, plan = buf.dispatch(x, None, topk, tpe, zero_copy=True)
    w = (torch.randn(E + 1, H, H, device="cuda") * 0.05).to(torch.bfloat16)
    done = torch.zeros(rows.shape[0] // 128 + 1, dtype=torch.int32, device="cuda")
    y = grouped_gemm(rows, w, cu, hooks=buf.gemm_hooks(done_counter=done))
    out, _, _ = buf.combine(plan, y, None, ready=(done, 4 * (H // 256)))
    buf.synchronize()
    want, _, _ = buf.combine(plan, y, None)
    assert torch.equal(out, want) and bool((done[: int(cu[-1]) // 128] == 4).all())
    be.set_timeout_ms(100)
    buf.combine(plan, y, None, ready=(done, 4 * (H // 256) + 1))
    with pytest.raises(MoonEPTimeoutError):
        buf.synchronize()
    assert torch.equal(buf.combine(plan, y, None)[0], want)
    buf.synchronize()
    buf.destroy()


def test_counts_that_do_not_match_the_routing():
    """More rows counted than routed: the rows nothing lands in are marked unused.  Fewer, or an expert that does not
    exist: an index error, and the Buffer works again afterwards."""
    S, H, K, E = 200, 64, 2, 6
    buf = Buffer(S, H, K, E, 1, token_padding=8)
    x, topk, tpe = _inputs(S, H, K, E, 0)
    buf._require_ctx()["hidden_buf_local"].fill_(7.0)
    rows, _, _, plan = buf.dispatch(x, None, topk, tpe + torch.tensor([0, 3, 0, 0, 0, 1], dtype=torch.int32, device="cuda"))
    buf.synchronize()
    assert torch.equal(rows, buf._require_ctx()["hidden_buf_local"])
    assert int((plan.src_info >= 0).sum()) == S * K
    for bad_topk, bad_tpe in ((topk, tpe - (tpe > 0).int()), (torch.where(topk == 2, E, topk), tpe)):
        buf.dispatch(x, None, bad_topk.contiguous(), bad_tpe)
        with pytest.raises(MoonEPIndexError):
            buf.synchronize()
    rows, _, _, plan = buf.dispatch(x, None, topk, tpe)
    buf.synchronize()
    assert torch.equal(buf.combine(plan, rows)[0], (x.float() * K).to(torch.bfloat16))
    buf.destroy()


@pytest.mark.parametrize("S", [1, 128, 129, 400])
def test_layer_forward_on_each_side_of_the_pair_rule(S):
    """One rank: up to 128 rows per expert the expert GEMMs run with one CTA per tile, above on CTA pairs."""
    from moonep_b200.models.moe_layer import ExpertParallelMoE, dense_reference

    H, K, E, inter = 256, 2, 2, 256
    buf = Buffer(S, H, K, E, 1, token_padding=128)
    layer = ExpertParallelMoE(buf, inter, init_std=0.05, seed=4)
    x, topk, tpe = _inputs(S, H, K, E, 0)
    gates = torch.rand(S, K, device="cuda")
    for save in (False, True):
        out, _ = layer.forward(x, gates, topk, tpe, save_for_backward=save)
        layer.check()
        ref = dense_reference(x.float().cpu(), gates.cpu(), topk.cpu(), *(w[:E].float().cpu() for w in (layer.w_gate, layer.w_up, layer.w_down)))
        # bf16 roundings of h, of every row and of the sum, each 2^-9 of values no larger than twice the largest result
        assert float((out.float().cpu() - ref).abs().max()) <= 8 * 2.0**-9 * float(ref.abs().max())
    layer.destroy()
    buf.destroy()


@pytest.mark.parametrize("sms", [None, 1, 3])
@pytest.mark.parametrize("S,H,K", [(40001, 8, 1), (9999, 264, 1), (301, 264, 1), (9999, 520, 2), (150, 2056, 2), (9999, 264, 3),
                                   (5001, 520, 4), (77, 520, 4), (301, 264, 5), (70, 265, 3), (40, 13, 9)])  # fmt: skip
def test_combine_with_one_to_eight_pieces_of_rows_in_hand(S, H, K, sms, monkeypatch):
    """The combine holds 8, 4, 2 or 1 pieces of 256 elements per warp by K and size, on a grid that is bounded or not:
    fp32 sums in ascending k rounded once, a lone row bit for bit (a negative zero and a NaN among its elements)."""
    if sms is not None:
        monkeypatch.setenv("MOONEP_LOCAL_SMS", str(sms))
    E = max(K, 4)
    buf = Buffer(S, H, K, E, 1, token_padding=4)
    x, topk, tpe = _inputs(S, H, K, E, 0)
    gates = torch.rand(S, K, device="cuda")
    rows, w, _, plan = buf.dispatch(x, gates, topk, tpe, zero_copy=True)
    loff = torch.where(plan.dst < 0, -plan.dst - 1, plan.dst).long().view(S, K)
    assert torch.equal(rows[loff.flatten()], x.repeat_interleave(K, 0))
    y = torch.randn(buf._require_ctx()["NvS"], H, generator=torch.Generator(device="cuda").manual_seed(K), device="cuda")
    y = y.to(torch.bfloat16)
    y[:, 0], y[loff[0], -1] = -0.0, float("nan")
    for with_weights in (True, False):
        out, back, _ = buf.combine(plan, y, w if with_weights else None)
        want = torch.zeros(S, H, device="cuda")
        for k in range(K):
            want += y[loff[:, k]].float()
        want = y[loff[:, 0]] if K == 1 else want.to(torch.bfloat16)
        same = (out.view(torch.int16) == want.view(torch.int16)) | (out.isnan() & want.isnan() & (K > 1))
        assert bool(same.all()) and (back is None or torch.equal(back, gates))
    buf.synchronize()
    buf.destroy()


def test_phases_of_the_dispatch_are_reported():
    S, H, K, E = 300, 512, 4, 8
    buf = Buffer(S, H, K, E, 1, token_padding=16)
    x, topk, tpe = _inputs(S, H, K, E, 0)
    _, _, _, plan = buf.dispatch(x, None, topk, tpe)
    be = buf._require_ctx()["_backend"]
    for args, names in (((x, None, topk, tpe), {"tables", "tokens", "send", "zero_fill", "build_expand"}),
                        ((x, None, None, None, plan), {"send", "zero_fill", "build_expand"})):  # fmt: skip
        be.reset_wait_stats()
        buf.dispatch(*args)
        buf.synchronize()
        phases = buf.stats()["kernel_phase_max_us"]
        assert set(phases) == names
    buf.destroy()


@pytest.mark.parametrize("S", [64, 400])
@pytest.mark.parametrize("switch", [None, "0", "1"])
def test_layer_reports_groups_that_are_not_whole_row_blocks(S, switch, monkeypatch):
    """The expert GEMMs take whole blocks of 128 rows.  A smaller padding works where the counts happen to fill them and is
    an index error otherwise, on one CTA per tile, on pairs and without hand-offs."""
    from moonep_b200.models.moe_layer import ExpertParallelMoE, dense_reference

    if switch is not None:
        monkeypatch.setenv("MOONEP_GEMM_PAIR", switch)
    H, E, inter = 256, 2, 256
    for K, rows, ok in ((1, 128, True), (2, S, False)):
        n = E * rows if ok else S
        buf = Buffer(n, H, K, E, 1, token_padding=16 if not ok else 64)
        layer = ExpertParallelMoE(buf, inter, init_std=0.05, seed=4)
        topk = ((torch.arange(n, device="cuda")[:, None] + torch.arange(K, device="cuda")) % E).to(torch.int32)
        tpe = torch.bincount(topk.flatten().long(), minlength=E).to(torch.int32)
        x = torch.randn(n, H, generator=torch.Generator(device="cuda").manual_seed(S), device="cuda").to(torch.bfloat16)
        gates = torch.ones(n, K, device="cuda")
        out, _ = layer.forward(x, gates, topk, tpe, save_for_backward=False)
        if ok:
            layer.check()
            ref = dense_reference(x.float().cpu(), gates.cpu(), topk.cpu(), *(w[:E].float().cpu() for w in (layer.w_gate, layer.w_up, layer.w_down)))
            # bf16 roundings of h, of every row and of the sum, each 2^-9 of values no larger than twice the largest result
            assert float((out.float().cpu() - ref).abs().max()) <= 8 * 2.0**-9 * float(ref.abs().max())
        else:
            with pytest.raises(MoonEPIndexError):
                layer.check()
        layer.destroy()
        buf.destroy()


@pytest.mark.parametrize("general", [False, True], ids=["single", "general"])
def test_layer_refuses_counts_above_what_was_routed(general, monkeypatch):
    """Rows of a group in which nothing landed would enter the weight gradients: an error in the layer (the general kernels'
    products wait for such rows in vain), although ``Buffer.dispatch`` takes such counts; the layer works again after it."""
    from moonep_b200.models.moe_layer import ExpertParallelMoE, dense_reference

    if general:
        monkeypatch.setenv("MOONEP_LOCAL_ROWS", "0")
        monkeypatch.setenv("MOONEP_TIMEOUT_MS", "200")
    S, H, K, E, inter = 200, 256, 2, 4, 256
    buf = Buffer(S, H, K, E, 1, token_padding=128)
    layer = ExpertParallelMoE(buf, inter, init_std=0.05, seed=4)
    x, topk, tpe = _inputs(S, H, K, E, 0)
    gates = torch.rand(S, K, device="cuda")
    for extra in (3, 128):
        more = tpe + torch.tensor([0, extra, 0, 0], dtype=torch.int32, device="cuda")
        for save in (False, True):
            layer.forward(x, gates, topk, more, save_for_backward=save)
            with pytest.raises(MoonEPTimeoutError if general else MoonEPIndexError):
                layer.check()
    buf.dispatch(x, gates, topk, more)
    buf.synchronize()
    out, saved = layer.forward(x, gates, topk, tpe)
    layer.check()
    ref = dense_reference(x.float().cpu(), gates.cpu(), topk.cpu(), *(w[:E].float().cpu() for w in (layer.w_gate, layer.w_up, layer.w_down)))
    # bf16 roundings of h, of every row and of the sum, each 2^-9 of values no larger than twice the largest result
    assert float((out.float().cpu() - ref).abs().max()) <= 8 * 2.0**-9 * float(ref.abs().max())
    layer.backward(saved, x)
    layer.check()
    layer.destroy()
    buf.destroy()
