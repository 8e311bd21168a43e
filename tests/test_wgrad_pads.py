"""Weight gradients leave out the rows of padding that a plan names: the same sums, bit for bit, with groups of one row, whole
groups, empty ones, and ranges that do not fit the groups."""

import pytest
import torch

from moonep_b200.ops.grouped_gemm import grouped_wgrad_rows


@pytest.mark.gpu
@pytest.mark.parametrize("per_group", [1, 4096])  # one CTA per tile, pairs
@pytest.mark.parametrize("used,step", [([1, 128, 0, 127, 16, 65], 128), ([700, 64, 129], 128), ([15, 0, 17, 33], 16)])
def test_pads_are_left_out(used, step, per_group):
    G, P, Q = len(used), 128, 256
    ends = torch.tensor([-(-n // step) * step for n in used]).cumsum(0)
    rows = int(ends[-1]) // 64 * 64 + 64
    g = torch.Generator().manual_seed(G)
    left, right = (torch.zeros(rows, n, dtype=torch.bfloat16) for n in (P, Q))
    pads, start = torch.zeros(G, 2, dtype=torch.int32), 0
    for i, (n, end) in enumerate(zip(used, ends.tolist())):
        left[start : start + n] = torch.randn(n, P, generator=g).bfloat16()
        right[start : start + n] = torch.randn(n, Q, generator=g).bfloat16()
        if end > start + n:
            pads[i] = torch.tensor([start + n, end - start - n])
        start = end
    left, right, cu, pads = left.cuda(), right.cuda(), ends.int().cuda(), pads.cuda()
    flags = torch.zeros(G, dtype=torch.int32, device="cuda")
    status = torch.zeros(8, dtype=torch.int32, device="cuda")
    wrong = pads.clone()
    wrong[:, 0] -= 16  # ranges that end before their groups are not believed
    got = []
    for ranges in (None, pads, wrong):
        out = torch.full((G, P, Q), 3.0, device="cuda")
        ptrs = torch.tensor([out[i].data_ptr() for i in range(G)], dtype=torch.int64, device="cuda")
        grouped_wgrad_rows(left, right, cu, ptrs, flags, status=status, rows_per_group=per_group, pads=ranges)
        got.append(out)
    assert int(status[0]) == 0 and torch.equal(got[0], got[1]) and torch.equal(got[0], got[2])
