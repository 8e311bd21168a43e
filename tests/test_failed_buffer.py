"""Kernels of a Buffer that has failed, or fails while they start.  Of a prefetch, slots keep what they held or get their
expert, nothing else is written, and after ``check_status`` the Buffer prefetches as before."""

import dataclasses
import re
import time

import pytest
import torch

from moonep_b200 import Buffer
from moonep_b200.constants import STATUS_BAD_INDEX
from moonep_b200.errors import MoonEPIndexError
from moonep_b200.models.routing import make_routing
from moonep_b200.ops._lib import CSRC
from moonep_b200.ops.grouped_gemm import grouped_gemm
from moonep_b200.parallel.world import LocalWorld


def _block(text, start):
    """From ``start`` to the end of the braces that are open there."""
    depth = 1
    for i in range(start, len(text)):
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        if depth == 0:
            return text[start:i]
    raise AssertionError("braces")


def test_threads_that_share_something_look_at_the_status_together():
    """The status word can change between two threads' looks at it.  Where every thread goes by its own look, none may wait for
    another in a barrier, or for what others write to shared memory."""
    leaves = re.compile(r"if \((?:poisoned\(c\)|failed != 0)\) return;|= !poisoned\(c\);")  # what follows in the function counts
    enters = re.compile(r"\bif \(.*!poisoned\(c\)\) \{")  # what is in the block counts
    shared = re.compile(r"__syncthreads|__shared__|bar\.sync")
    seen = 0
    for path in sorted(CSRC.glob("*.cu")):
        text = path.read_text()
        parts = [text[m.end() : text.index("\n}\n", m.end())] for m in leaves.finditer(text)]
        parts += [_block(text, m.end()) for m in enters.finditer(text)]
        seen += len(parts)
        assert not any(shared.search(part) for part in parts), f"{path.name}: threads share something, but each by its own look"
    assert seen


@pytest.mark.gpu
@pytest.mark.parametrize("B,num_sms", [(3, 5), (40, 148)])
def test_prefetch_on_a_failed_buffer(B, num_sms):
    S, H, K, epn, R, Hw, Hp = 32, 64, 2, 4, 2, 256, 384
    E, lw = R * epn, LocalWorld(R, "cuda")
    bufs = lw.run(lambda r: Buffer(S, H, K, E, R, num_sms=num_sms, token_padding=8, B=B, world=lw.view(r)))
    table = (torch.arange(R * B, dtype=torch.int32).view(R, B) * 3 % (E + 1) - 1).cuda()  # slots without an expert among them
    empty = torch.full((B, Hw, Hp), -123.0, dtype=torch.bfloat16, device="cuda")
    experts = [torch.randn(E, Hw, Hp, generator=torch.Generator(device="cuda").manual_seed(t), device="cuda").bfloat16() for t in range(3)]
    sms, side = torch.cuda.get_device_properties(0).multi_processor_count, torch.cuda.Stream()
    rows, weights = torch.zeros(128 * sms, 4096, device="cuda").bfloat16(), torch.zeros(1, 16384, 4096, device="cuda").bfloat16()
    ends = torch.tensor([128 * sms], dtype=torch.int32, device="cuda")
    wants = [[torch.where(row[:, None, None] >= 0, e[row.long().clamp(min=0)], empty) for e in experts] for row in table]

    def body(r):
        buf = bufs[r]
        be = buf._require_ctx()["_backend"]
        topk, tpe, gates = make_routing("biased", S, K, E, R, r, bias=1.5, seed=5, device="cuda")
        plan = buf.dispatch(torch.ones(S, H, device="cuda").bfloat16(), gates, topk, tpe)[3]

        def fetch(etc, late=False):
            full = [torch.cat([e, empty]).contiguous() for e in experts]
            if late:  # most CTAs of the prefetch have to wait for an SM, and start when the first one has seen the table
                side.wait_stream(torch.cuda.current_stream())
                with torch.cuda.stream(side):
                    grouped_gemm(rows, weights, ends, num_sms=sms - 8, pair=False)
                time.sleep(0.0003)
            buf.prefetch_weight(dataclasses.replace(plan, experts_to_copy=etc), full_gate_weight=full[0], full_up_weight=full[1],
                                full_down_weight=full[2])  # fmt: skip
            torch.cuda.synchronize()
            assert all(torch.equal(f[:E], e) for f, e in zip(full, experts))
            return [f[E:] for f in full]

        def whole():
            got = fetch(table)
            buf.check_status()
            return all(torch.equal(g, w) for g, w in zip(got, wants[r]))

        def failed(etc, late=False):
            got = fetch(etc, late)
            with pytest.raises(MoonEPIndexError):
                buf.check_status()
            # pieces counted towards slots that were not finished would announce the next prefetch's slots too early
            assert not bool(be._slot_scratch()[1].any())
            return got

        assert whole()
        be.status[0] = STATUS_BAD_INDEX  # before the kernel starts: no slot is written
        assert all(torch.equal(g, empty) for g in failed(table))
        assert whole()
        for late in (False, True, True):  # while it starts: the first CTA meets an expert that is none
            bad = table.clone()
            bad[r, B - 1] = E
            for g, w in zip(failed(bad, late), wants[r]):
                assert torch.equal(g[B - 1], empty[0])
                assert bool(((g[:-1] == w[:-1]) | (g[:-1] == empty[:-1])).all())
            assert whole()

    lw.run(body)
    lw.run(lambda r: bufs[r].destroy())
