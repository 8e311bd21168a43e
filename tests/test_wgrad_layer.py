"""Weight gradients of several weights in one launch are those of a launch each, bit for bit."""

import pytest
import torch

from moonep_b200.ops.grouped_gemm import grouped_wgrad_layer, grouped_wgrad_rows


@pytest.mark.gpu
@pytest.mark.parametrize("per_group", [128, 1024])  # one CTA per tile, and pairs
# one group and many, empty ones, an odd number of 128-column tiles, one weight, two and three of different shapes
@pytest.mark.parametrize("rows,shapes", [([128], [(128, 256)]), ([256, 0, 128], [(384, 512), (512, 256)]), ([1024] * 5, [(256, 512), (512, 256), (128, 768)]),
                                         ([128] * 40, [(256, 256)] * 3), ([0, 0], [(128, 256), (256, 256)])])  # fmt: skip
def test_one_launch_gives_what_one_each_gives(rows, shapes, per_group):
    g = torch.Generator(device="cuda").manual_seed(sum(rows) + len(shapes))
    cu = torch.tensor(rows).cumsum(0).int().cuda()
    G, n, status = len(rows), max(64, sum(rows)), torch.zeros(8, dtype=torch.int32, device="cuda")
    ops = [tuple(torch.randn(n, c, generator=g, device="cuda").bfloat16() for c in pq) for pq in shapes]
    flags = torch.tensor([i % 3 for i in range(G)], dtype=torch.int32, device="cuda")  # store, add, leave alone if empty
    got = []
    for together in (True, False):
        outs = [torch.full((G, P, Q), 2.0, device="cuda") for P, Q in shapes]
        # the last weight's second group has no target
        ptrs = [[0 if G > 1 and g == 1 and rows[1] == 0 and i == len(shapes) - 1 else o[g].data_ptr() for g in range(G)] for i, o in enumerate(outs)]
        weights = [(l, r, torch.tensor(p, dtype=torch.int64).cuda()) for (l, r), p in zip(ops, ptrs)]
        if together:
            grouped_wgrad_layer(weights, cu, flags, status=status, rows_per_group=per_group)
        else:
            for l, r, p in weights:
                grouped_wgrad_rows(l, r, cu, p, flags, status=status, rows_per_group=per_group)
        got.append(outs)
    assert all(torch.equal(a, b) for a, b in zip(*got))
    assert int(status[0]) == 0
    for (l, r), out in zip(ops, got[0]):
        want = l[: rows[0]].double().T @ r[: rows[0]].double()
        # fp32 sums of exact products: at most `rows` additions, each rounded to 2^-24 of a partial sum
        bound = l[: rows[0]].double().abs().T @ r[: rows[0]].double().abs() * (rows[0] + 2) * 2.0**-24
        assert bool(((out[0].double() - want).abs() <= bound).all())
