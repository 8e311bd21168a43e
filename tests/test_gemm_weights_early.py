"""A GEMM that asks for its weights while the GEMM before it on the stream still runs reads that GEMM's output only once it is
whole: the same sums, bit for bit, as one that waits first."""

import pytest
import torch

from moonep_b200.ops.grouped_gemm import grouped_gemm


@pytest.mark.gpu
# fewer K blocks than stages, as many and more; one tile per CTA, some CTAs without one, more than one; cut tiles; no rows
@pytest.mark.parametrize("rows,H,I", [([128] * 3, 256, 128), ([128, 0, 256], 256, 256), ([128] * 16, 2048, 1024), ([128, 384] * 10, 512, 512),
                                      ([128] * 148, 1024, 256), ([128] * 8, 4096, 512), ([0, 0], 256, 128)])  # fmt: skip
def test_weights_before_rows(rows, H, I):
    g = torch.Generator(device="cuda").manual_seed(H + I)
    cu = torch.tensor(rows).cumsum(0).int().cuda()
    n, cap, G = int(cu[-1]), int(cu[-1]) + 128, len(rows)
    gate, up = ((torch.randn(G, I, H, generator=g, device="cuda") * H**-0.5).bfloat16() for _ in range(2))
    down = (torch.randn(G, H, I, generator=g, device="cuda") * I**-0.5).bfloat16()
    scale, status = torch.rand(cap, generator=g, device="cuda"), torch.zeros(8, dtype=torch.int32, device="cuda")
    xs = [torch.randn(cap, H, generator=g, device="cuda").bfloat16() for _ in range(3)]
    h = torch.zeros(cap, I, device="cuda").bfloat16()  # the same for every pass: a row read too soon is another pass's

    def passes(early):
        outs = []
        for i in range(9):
            grouped_gemm(xs[i % 3], gate, cu, w_up=up, mode="swiglu", out=h, status=status, pair=False)
            outs.append(grouped_gemm(h, down, cu, mode="scale", row_scale=scale, status=status, pair=False, weights_early=early)[:n])
        return outs

    assert all(torch.equal(a, b) for a, b in zip(passes(True), passes(False)))
    assert int(status[0]) == 0
