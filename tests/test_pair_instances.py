"""The CTA-pair GEMM's instances (stages, epilogue warps) on both sides of every line of its dispatch, with pad rows of zeros,
groups of one, two and three row blocks and a last block that ends where the tensor does; against fp32 products."""

import pytest
import torch

from moonep_b200.ops.grouped_gemm import grouped_gemm, grouped_gemm_kn
from tests.test_grouped_gemm import ACC_REL, _abs_dot, _assert_elementwise, grouped_gemm_reference_fp32

pytestmark = pytest.mark.gpu


def _inputs(K, N):
    g = torch.Generator().manual_seed(K)
    rows = [128, 0, 384, 256]
    cu = torch.tensor(rows).cumsum(0).to(torch.int32).cuda()
    total = sum(rows)
    x = (torch.randn(total, K, generator=g) * 0.5).to(torch.bfloat16).cuda()
    x[100:128] = 0  # pad rows at groups' ends
    x[-64:] = 0
    w, w2 = ((torch.randn(4, N, K, generator=g) * 0.05).to(torch.bfloat16).cuda() for _ in range(2))
    return x, w, w2, cu, torch.rand(total, generator=g).cuda(), total


@pytest.mark.parametrize("K", [448, 512, 1024, 1088, 2048, 2112])
def test_instances_match_fp32_products(K):
    N = 256
    x, w, w2, cu, scale, total = _inputs(K, N)
    a, u = grouped_gemm_reference_fp32(x, w, cu), grouped_gemm_reference_fp32(x, w2, cu)
    da, du = _abs_dot(x, w, cu, total), _abs_dot(x, w2, cu, total)
    _assert_elementwise(grouped_gemm(x, w, cu, pair=True).float(), a, da, "plain")
    _assert_elementwise(grouped_gemm(x, w, cu, row_scale=scale, mode="scale", pair=True).float(), a * scale[:, None],
                        da * scale[:, None], "scale")
    kn = grouped_gemm_kn(x, [w.transpose(1, 2).contiguous()], cu)
    _assert_elementwise(kn.float(), a, da, "[K, N]")
    h = torch.nn.functional.silu(a) * u
    # |silu(a)| <= |a| and its slope is below 1.1, so errors of a and u of ACC_REL * d reach h by at most this
    slack = 1.1 * da * u.abs() + du * torch.nn.functional.silu(a).abs() + ACC_REL * 1.1 * da * du
    pre = tuple(torch.full((total, N), 7.0, dtype=torch.bfloat16, device="cuda") for _ in range(2))
    # __expf and the division add a few 2^-22 of h, far inside one of the two 2^-9 that BF16_REL leaves
    for got in (grouped_gemm(x, w, cu, w_up=w2, mode="swiglu", pair=True),
                grouped_gemm(x, w, cu, w_up=w2, mode="swiglu", pair=True, save_pre=pre),
                grouped_gemm(x, w, cu, w_up=w2, mode="swiglu", pair=False)):  # fmt: skip
        _assert_elementwise(got.float(), h, slack, "SwiGLU")
        assert not got[100:128].any() and not got[-64:].any(), "rows of zeros"
    _assert_elementwise(pre[0].float(), a, da, "pre-activation of the gate")
    _assert_elementwise(pre[1].float(), u, du, "pre-activation of the up projection")
