"""Workloads of the library for timing: what they are (``listed``, ``draw``), their inputs (``prepare``), one pass
through the public API (``run``), the work such a pass cannot do without (``work``) and what it has to give
(``tolerance``, ``exact``).  One GPU; every pass goes through ``Buffer``, ``ExpertParallelMoE``, ``MoEBlock`` and
``ExpertAdamW`` as a program that uses the library calls them.

Kinds of case
-------------
exchange   ``Buffer.dispatch`` + ``Buffer.combine`` of one rank: a fresh plan (forward direction), a replayed plan
           (backward direction) or a captured CUDA graph; zero-copy or staged; any padding, with or without weights
emulated   the same operations with ``prefetch_weight`` and ``reduce_grad`` on several ranks of one process, which is
           how the multi-rank paths run where there is one GPU
layer      ``ExpertParallelMoE``: inference (forward only) or a training step (forward, backward, SGD)
block      ``MoEBlock`` with autograd and ``ExpertAdamW``: router, experts, backward, optimizer step
"""

from __future__ import annotations

import math

import torch

from moonep_b200 import Buffer
from moonep_b200.models.moe_block import MoEBlock
from moonep_b200.models.moe_layer import ExpertParallelMoE
from moonep_b200.models.optim import ExpertAdamW
from moonep_b200.parallel.symm import create_full_expert_weight, create_nvl_dist_tensor, view_nvl_dist_rows
from moonep_b200.parallel.world import LocalWorld

LR = 1e-5


def _exchange(name, S, H, K, E, **kw):
    case = {"kind": "exchange", "S": S, "H": H, "K": K, "E": E, "pad": 128, "routing": "softmax", "mode": "fresh",
            "zero_copy": True, "weights": True}  # fmt: skip
    case.update(kw)
    return case if name is None else {"name": name, **case}


def _emulated(name, R, S, H, K, E, inter, **kw):
    case = {"kind": "emulated", "R": R, "S": S, "H": H, "K": K, "E": E, "I": inter, "pad": 128, "routing": "zipf"}
    case.update(kw)
    return case if name is None else {"name": name, **case}


def _layer(name, S, H, K, E, inter, train):
    case = {"kind": "layer", "S": S, "H": H, "K": K, "E": E, "I": inter, "train": train}
    return case if name is None else {"name": name, **case}


def _block(name, S, H, K, E, inter):
    case = {"kind": "block", "S": S, "H": H, "K": K, "E": E, "I": inter}
    return case if name is None else {"name": name, **case}


def listed():
    return [
        # one decode step of a small batch, replayed as a CUDA graph: latency of the kernels alone
        _exchange("decode_graph_s16", 16, 7168, 8, 256, mode="graph"),
        # the smallest size of the token sweep, called eagerly: launches and host work count
        _exchange("exchange_s128", 128, 7168, 8, 256),
        # the headline benchmark of the repository on one rank
        _exchange("exchange_s4096", 4096, 7168, 8, 256),
        # the largest size of the token sweep: a long prefill or a large training batch
        _exchange("exchange_s16384", 16384, 7168, 8, 256),
        # the skewed-routing benchmark, through the copying (non zero-copy) calls with an expert output of its own
        _exchange("skew_staged_s8192", 8192, 4096, 6, 64, routing="zipf", zero_copy=False),
        # ragged sizes: nothing is a power of two, rows are 16-byte but not 128-byte multiples, small padding
        _exchange("ragged_s1777", 1777, 2056, 5, 24, pad=16),
        # the backward direction: a plan is replayed for the gradients, which carry no gate weights out
        _exchange("replay_s2048", 2048, 4096, 8, 128, mode="replay", weights=False),
        # the multi-rank operations with hot experts, their weights and gradients, two ranks in one process
        _emulated("two_ranks_s4096", 2, 4096, 7168, 8, 64, 256),
        # serving: one decode batch through the expert layer (weights bound it), and a prefill (tensor cores bound it)
        _layer("layer_decode_s64", 64, 2048, 4, 16, 1024, False),
        _layer("layer_prefill_s4096", 4096, 4096, 4, 16, 1024, False),
        # training: the layer benchmark's hidden and intermediate sizes and rows per expert, with fewer experts
        _layer("layer_train_s2048", 2048, 7168, 4, 8, 2048, True),
        # a training program: router, autograd and Adam around a layer of moderate size
        _block("block_train_s2048", 2048, 2048, 4, 16, 1024),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["exchange"] * 5 + ["emulated", "layer", "layer", "block"])
    if kind == "exchange":
        S, K = _log_int(rng, 1, 16384), rng.randint(1, 12)
        H = 8 * _log_int(rng, 32, 1024)
        E = rng.randint(max(K, 4), 256)
        while S * K * H > 16384 * 8 * 7168:
            S = (S + 1) // 2
        mode = rng.choice(["fresh", "fresh", "replay", "graph"])
        return _exchange(None, S, H, K, E, pad=rng.choice([1, 8, 16, 64, 128, 128]), mode=mode,
                         routing=rng.choice(["softmax", "zipf"]), zero_copy=mode == "graph" or rng.random() < 0.7,
                         weights=mode != "replay" and rng.random() < 0.8)  # fmt: skip
    if kind == "emulated":
        R = rng.choice([2, 2, 4])
        E = R * rng.randint(4, 64 // R)
        return _emulated(None, R, _log_int(rng, 32, 8192 // R), 128 * rng.randint(2, 56), rng.randint(1, 6), E,
                         128 * rng.randint(1, 2), routing=rng.choice(["softmax", "zipf"]))  # fmt: skip
    E = rng.randint(4, 16)
    S, H, K, inter = _log_int(rng, 32, 4096), 256 * rng.randint(2, 16), rng.randint(1, 4), 256 * rng.randint(1, 4)
    if kind == "layer":
        return _layer(None, S, H, K, E, inter, rng.random() < 0.5)
    return _block(None, min(S, 2048), min(H, 2048), K, E, inter)


# -- inputs ---------------------------------------------------------------------------------------------------------


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _tokens(S, H, gen, scale=1.0):
    return (torch.randn(S, H, generator=gen, device="cuda") * scale).to(torch.bfloat16)


def _routing(pattern, S, K, E, gen, shared=None):
    """Top-k experts, softmax gates and token counts: router logits ~ N(0,1), or experts drawn without replacement by
    a Zipf(1.2) popularity over a random permutation (``shared``: the generator of that permutation)."""
    noise = torch.rand(S, E, generator=gen, device="cuda").clamp_(1e-20, 1 - 1e-7)
    if pattern == "zipf":
        pop = torch.arange(1, E + 1, device="cuda", dtype=torch.float32) ** -1.2
        pop = pop[torch.randperm(E, generator=shared or gen, device="cuda")]
        logits = pop.log() - (-noise.log()).log()  # Gumbel top-k: draws without replacement
        gates_from = torch.randn(S, K, generator=gen, device="cuda")
    else:
        logits = torch.randn(S, E, generator=gen, device="cuda")
        gates_from = None
    top, topk = torch.topk(logits, K, dim=1)
    gates = torch.softmax(top if gates_from is None else gates_from, dim=1)
    topk = topk.to(torch.int32).contiguous()
    return topk, gates.contiguous(), torch.bincount(topk.flatten().long(), minlength=E).to(torch.int32)


def prepare(case, seed):
    return _PREPARE[case["kind"]](case, seed)


def _prepare_exchange(c, seed):
    S, H, K, E, gen = c["S"], c["H"], c["K"], c["E"], _gen(seed)
    buf = Buffer(S, H, K, E, 1, num_sms=32, token_padding=c["pad"])
    topk, gates, tpe = _routing(c["routing"], S, K, E, gen)
    st = {"case": c, "buf": buf, "x": _tokens(S, H, gen), "gates": gates if c["weights"] else None, "topk": topk, "tpe": tpe}
    if not c["zero_copy"]:  # what the experts made of the rows
        nvs = S * K + 2 * E * (c["pad"] - 1)
        st["y"] = _tokens(nvs, H, gen)
        st["y_w"] = torch.rand(nvs, generator=gen, device="cuda") if c["weights"] else None
    if c["mode"] == "replay":
        st["plan"] = buf.dispatch(st["x"], gates, topk, tpe)[3]
    if c["mode"] == "graph":
        st["step"] = buf.capture(lambda: _round_trip(st))
    return st


def _prepare_emulated(c, seed):
    R, S, H, K, E, inter = c["R"], c["S"], c["H"], c["K"], c["E"], c["I"]
    world, epn, gen = LocalWorld(R, "cuda:0"), E // R, _gen(seed)
    shapes = ((inter, H), (inter, H), (H, inter))
    experts = [(torch.randn(E, a, b, generator=gen, device="cuda") * 0.02).to(torch.bfloat16) for a, b in shapes]
    sent = [[torch.randn(epn, a, b, generator=gen, device="cuda") for a, b in shapes] for _ in range(R)]
    perm_seed = 7919 + int(seed)

    def make(r):
        v, gr = world.view(r), _gen(int(seed) * 1009 + r + 1)
        topk, gates, tpe = _routing(c["routing"], S, K, E, gr, _gen(perm_seed))
        ws = [create_full_expert_weight(E, epn, a, b, v) for a, b in shapes]
        for w, e in zip(ws, experts):
            w[:E].copy_(e)
        red = [view_nvl_dist_rows(create_nvl_dist_tensor([epn, a, b], torch.float32, v, pad_dim0=False), R, epn)
               for a, b in shapes]  # fmt: skip
        for t, g in zip(red, sent[r]):
            t[r].copy_(g)
        return {"buf": Buffer(S, H, K, E, R, num_sms=32, token_padding=c["pad"], world=v), "x": _tokens(S, H, gr),
                "topk": topk, "gates": gates, "tpe": tpe, "w": ws, "red": red,
                "grad": [torch.zeros(epn, a, b, device="cuda") for a, b in shapes]}  # fmt: skip

    return {"case": c, "world": world, "ranks": world.run(make)}


def _prepare_layer(c, seed):
    S, H, K, E, gen = c["S"], c["H"], c["K"], c["E"], _gen(seed)
    buf = Buffer(S, H, K, E, 1, num_sms=32, token_padding=128)
    block = c["kind"] == "block"
    net = (MoEBlock if block else ExpertParallelMoE)(buf, c["I"], init_std=0.02, seed=int(seed) % 100003)
    st = {"case": c, "buf": buf, "net": net, "x": _tokens(S, H, gen), "go": _tokens(S, H, gen, 0.1)}
    if block:
        st["x"].requires_grad_(True)
        st["opt"] = ExpertAdamW(net.experts, lr=LR, weight_decay=0.1)
    else:
        st["topk"], st["gates"], st["tpe"] = _routing("softmax", S, K, E, gen)
    return st


_PREPARE = {"exchange": _prepare_exchange, "emulated": _prepare_emulated, "layer": _prepare_layer, "block": _prepare_layer}


# -- one pass -------------------------------------------------------------------------------------------------------


def run(st):
    return _RUN[st["case"]["kind"]](st)


def _round_trip(st):
    c, buf = st["case"], st["buf"]
    if c["mode"] == "replay":
        plan, cu = st["plan"], None
        xn, wn, _, _ = buf.dispatch(st["x"], st["gates"], plan=plan, zero_copy=c["zero_copy"])
    else:
        xn, wn, cu, plan = buf.dispatch(st["x"], st["gates"], st["topk"], st["tpe"], zero_copy=c["zero_copy"])
    y, yw = (xn, wn) if c["zero_copy"] else (st["y"], st["y_w"])
    out, back, _ = buf.combine(plan, y, yw, zero_copy=c["zero_copy"])
    return {"rows": xn, "row_weights": wn, "cu_seqlens": cu, "dst": plan.dst, "out": out, "gates": back}


def _run_exchange(st):
    return st["step"].replay() if "step" in st else _round_trip(st)


def _run_emulated(st):
    def body(r):
        s = st["ranks"][r]
        buf, E = s["buf"], st["case"]["E"]
        xn, wn, cu, plan = buf.dispatch(s["x"], s["gates"], s["topk"], s["tpe"], zero_copy=True)
        buf.prefetch_weight(plan, full_gate_weight=s["w"][0], full_up_weight=s["w"][1], full_down_weight=s["w"][2])
        out, back, _ = buf.combine(plan, xn, wn, zero_copy=True)
        buf.reduce_grad(plan, False, *s["grad"], *s["red"], owner_local=True)
        return {"out": out, "gates": back, "cu_seqlens": cu, "dst": plan.dst, "slots": [w[E:] for w in s["w"]],
                "grads": s["grad"]}  # fmt: skip

    return st["world"].run(body)


def _run_layer(st):
    layer = st["net"]
    out, saved = layer.forward(st["x"], st["gates"], st["topk"], st["tpe"], save_for_backward=st["case"]["train"])
    if not st["case"]["train"]:
        return {"out": out}
    dx, dgates = layer.backward(saved, st["go"])
    layer.sgd_step(LR)
    layer.zero_grad()
    return {"out": out, "dx": dx, "dgates": dgates, "grads": list(layer.owner_grads()), "weights": list(layer.owner_weights())}


def _run_block(st):
    net, x, opt = st["net"], st["x"], st["opt"]
    y = net(x)
    y.backward(st["go"])
    opt.step()
    opt.zero_grad()
    dx, dr = x.grad, net.router.weight.grad
    x.grad = net.router.weight.grad = None
    return {"out": y.detach(), "dx": dx, "router_grad": dr, "grads": list(net.experts.owner_grads()),
            "weights": list(net.experts.owner_weights()), "master": opt.master, "exp_avg": opt.exp_avg,
            "exp_avg_sq": opt.exp_avg_sq}  # fmt: skip


_RUN = {"exchange": _run_exchange, "emulated": _run_emulated, "layer": _run_layer, "block": _run_block}


# -- what a pass cannot do without ------------------------------------------------------------------------------------


def work(case):
    """Bytes: each input read and each output written once (the dispatched rows are an output and an input).  Rows of
    padding, whose number depends on the routing, count as half a group's padding for every expert in use."""
    S, H, K, E = case["S"], case["H"], case["K"], case["E"]
    rows, used = S * K, min(E, S * K)
    if case["kind"] == "exchange":
        pad = used * (case["pad"] - 1) // 2
        # tokens in, rows out and in again, results out; gates likewise, routing in, plan out
        return {"bytes": 2 * H * (2 * S + 2 * rows + pad) + 24 * rows, "flops": 0}
    if case["kind"] == "emulated":
        R, inter = case["R"], case["I"]
        pad = R * used * (case["pad"] - 1) // 2
        moved = 3 * E * inter * H // 8  # hot experts: about one slot in eight is in use
        return {"bytes": 2 * H * (R * (2 * S + 2 * rows) + pad) + moved * (4 + 12), "flops": 0}
    inter = case["I"]
    n = 3 * used * inter * H
    if case["kind"] == "layer" and not case["train"]:
        return {"bytes": 2 * n + 4 * S * H, "flops": 6 * rows * inter * H}
    n_all = 3 * E * inter * H
    # weights read by both directions, fp32 gradients out; SGD: gradients in, weights in and out; Adam: three fp32
    # states in and out, gradients in, weights out
    update = 4 + 2 + 2 if case["kind"] == "layer" else 24 + 4 + 2
    extra = 6 * S * E * H if case["kind"] == "block" else 0
    return {"bytes": 2 * 2 * n + 4 * n_all + update * n_all + 8 * S * H, "flops": 18 * rows * inter * H + extra}


def tolerance(case):
    if case["kind"] == "exchange" and case["zero_copy"]:
        return "exact"  # copies, and sums of at most 12 equal bf16 values, which 32 bits hold exactly
    if case["kind"] == "exchange":
        return {"rel": 2e-3, "max": 8e-3}  # one rounding to bf16 of a 32-bit sum
    if case["kind"] == "emulated":
        return {"rel": 4e-3, "max": 1.6e-2}  # two roundings to bf16: per rank, and of the ranks' sum
    return {"rel": 1e-2, "max": 0.5}  # chains of bf16 products; single values near zero differ by more than their size


# -- the same in 64 bits ----------------------------------------------------------------------------------------------


def exact(case, seed):
    return {"exchange": _exact_exchange, "emulated": _exact_emulated, "layer": _exact_layer, "block": _exact_layer}[
        case["kind"]](case, seed)  # fmt: skip


def _exact_exchange(c, seed):
    S, H, K, E, pad, gen = c["S"], c["H"], c["K"], c["E"], c["pad"], _gen(seed)
    topk, gates, tpe = _routing(c["routing"], S, K, E, gen)
    x = _tokens(S, H, gen)
    nvs = S * K + 2 * E * (pad - 1)
    flat, counts = topk.flatten().long(), tpe.long()
    padded = (counts + pad - 1) // pad * pad
    ends = padded.cumsum(0)
    order = torch.argsort(flat, stable=True)
    first = counts.cumsum(0) - counts
    loff = torch.empty_like(flat)
    loff[order] = torch.arange(S * K, device="cuda") - first[flat[order]] + (ends - padded)[flat[order]]
    rows = torch.zeros(nvs, H, dtype=torch.float64, device="cuda")
    rows[loff] = x.double().repeat_interleave(K, dim=0)
    if c["zero_copy"]:
        out, back = x.double() * K, gates.double()
    else:
        y = _tokens(nvs, H, gen)
        out = torch.zeros(S, H, dtype=torch.float64, device="cuda")
        for k in range(K):
            out += y[loff.view(S, K)[:, k]].double()
        back = torch.rand(nvs, generator=gen, device="cuda")[loff].view(S, K).double() if c["weights"] else None
    return {"rows": rows, "row_weights": None, "cu_seqlens": None,
            "dst": None, "out": out, "gates": back if c["weights"] else None}  # fmt: skip


def _exact_emulated(c, seed):
    got = []
    for r in range(c["R"]):
        gr = _gen(int(seed) * 1009 + r + 1)
        _, gates, _ = _routing(c["routing"], c["S"], c["K"], c["E"], gr, _gen(7919 + int(seed)))
        x = _tokens(c["S"], c["H"], gr)
        got.append({"out": x.double() * c["K"], "gates": gates.double(), "cu_seqlens": None, "dst": None, "slots": None,
                    "grads": None})  # fmt: skip
    return got


def _initial_weights(c, seed):
    """The experts' weights as the layer makes them (bf16, from the seed, one generator per weight and expert)."""
    made = []
    for t, (a, b) in enumerate(((c["I"], c["H"]), (c["I"], c["H"]), (c["H"], c["I"]))):
        of = [torch.randn(a, b, generator=torch.Generator().manual_seed((int(seed) % 100003) * 1_000_003 + t * 10_007 + e))
              for e in range(c["E"])]  # fmt: skip
        made.append(torch.stack([(w * 0.02).to(torch.bfloat16) for w in of]).cuda().double())
    return made


def _exact_layer(c, seed):
    S, H, K, E, gen = c["S"], c["H"], c["K"], c["E"], _gen(seed)
    ws = _initial_weights(c, seed)
    x, go = _tokens(S, H, gen).double(), _tokens(S, H, gen, 0.1).double()
    if c["kind"] == "layer" and not c["train"]:
        topk, gates, _ = _routing("softmax", S, K, E, gen)
        with torch.no_grad():
            return {"out": _experts(x, gates.double(), topk, ws, E)}
    for w in ws:
        w.requires_grad_(True)
    x.requires_grad_(True)
    if c["kind"] == "layer":
        topk, gates, _ = _routing("softmax", S, K, E, gen)
        gates = gates.double().requires_grad_(True)
        out = _experts(x, gates, topk, ws, E)
        out.backward(go)
        return {"out": out.detach(), "dx": x.grad, "dgates": gates.grad, "grads": [w.grad for w in ws],
                "weights": [w.detach() - LR * w.grad for w in ws]}  # fmt: skip
    rg = torch.Generator().manual_seed(int(seed) % 100003 + 17)
    wr = (torch.randn(E, H, generator=rg) * 0.02).cuda().double().requires_grad_(True)
    top, topk = torch.topk(torch.softmax(x @ wr.t(), dim=-1), K, dim=-1)
    out = _experts(x, top / top.sum(dim=-1, keepdim=True), topk, ws, E)
    out.backward(go)
    res = {"out": out.detach(), "dx": x.grad, "router_grad": wr.grad, "grads": [w.grad for w in ws]}
    b1, b2, eps = 0.9, 0.95, 1e-8
    new = [w.detach() * (1 - LR * 0.1) - LR * w.grad / (w.grad.abs() + eps) for w in ws]
    res.update(weights=new, master=new, exp_avg=[(1 - b1) * w.grad for w in ws], exp_avg_sq=[(1 - b2) * w.grad**2 for w in ws])
    return res


def _experts(x, gates, topk, ws, E):
    out = torch.zeros_like(x)
    for e in range(E):
        s, k = torch.where(topk == e)
        if s.numel():
            xe = x[s]
            h = torch.nn.functional.silu(xe @ ws[0][e].t()) * (xe @ ws[1][e].t())
            out = out.index_add(0, s, (h @ ws[2][e].t()) * gates[s, k][:, None])
    return out
