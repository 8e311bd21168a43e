"""Products with weights as stored on one CTA per tile: those of the CTA pairs, whole tiles and cut ones, weights asked for
early or not."""

import pytest
import torch

from moonep_b200.ops.grouped_gemm import grouped_gemm_kn, grouped_gemm_kn_reference


@pytest.mark.gpu
# quarters, halves and whole tiles; one weight and two; fewer and more K blocks than stages; empty groups; no rows
@pytest.mark.parametrize("rows,Ks,N", [([128], [64], 256), ([128, 0, 384], [128, 64], 768), ([128] * 37, [64], 256), ([128] * 38, [192], 256),
                                       ([128] * 74, [64], 256), ([128] * 75, [64], 256), ([256] * 4, [1152], 512),
                                       ([128, 128] * 9, [512, 704], 1024), ([0, 0], [64], 256)])  # fmt: skip
def test_kn_on_single_ctas(rows, Ks, N):
    g = torch.Generator(device="cuda").manual_seed(N + sum(rows))
    cu = torch.tensor(rows).cumsum(0).int().cuda()
    n, cap, K = int(cu[-1]), max(128, int(cu[-1])) + 128, sum(Ks)
    x = torch.randn(cap, K, generator=g, device="cuda").bfloat16()
    ws = [(torch.randn(len(rows), k, N, generator=g, device="cuda") * K**-0.5).bfloat16() for k in Ks]
    status = torch.zeros(8, dtype=torch.int32, device="cuda")
    got = []
    for kw in ({"pair": False}, {"pair": False, "weights_early": True}, {"pair": False, "num_sms": 2}, {"pair": True}):
        out = torch.full((cap, N), 3.0, device="cuda").bfloat16()
        grouped_gemm_kn(x, ws, cu, out=out, status=status, **kw)
        assert bool((out[n:] == 3.0).all()), kw
        got.append(out)
    assert all(torch.equal(got[0], o) for o in got[1:3])  # the order of a sum does not depend on the tile
    assert int(status[0]) == 0
    want = grouped_gemm_kn_reference(x, ws, cu)
    for o in got:  # fp32 sums of another order, each rounded to bf16: a step apart at most (2^-7 of the value), and their difference
        assert bool(((o[:n].float() - want[:n].float()).abs() <= 2.0**-7 * want[:n].float().abs() + 2e-3).all())
