"""Products of few row blocks are cut by columns into halves and quarters of tiles, as far as there are SMs for them: the same
sums, bit for bit, as the whole tiles that a bound on the SMs leaves, and the per-group reference's within rounding."""

import pytest
import torch

from moonep_b200.ops.grouped_gemm import grouped_gemm, grouped_gemm_reference


def _operands(rows, K, N, seed=0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    cu = torch.tensor(rows).cumsum(0).int().cuda()
    cap = max(128, int(cu[-1])) + 128
    x = torch.randn(cap, K, generator=g, device="cuda").bfloat16()
    w, up = ((torch.randn(len(rows), N, K, generator=g, device="cuda") * K**-0.5).bfloat16() for _ in range(2))
    return cu, x, w, up, torch.rand(cap, generator=g, device="cuda")


def _close(got, want):
    """Both round an fp32 sum of another order to bf16: a step apart at most (2^-7 of the value), and the sums' difference."""
    return bool(((got.float() - want.float()).abs() <= 2.0**-7 * want.float().abs() + 2e-3).all())


@pytest.mark.gpu
# whole tiles of a step: 4 (quarters), 37 and 38 (quarters of 148 SMs, and halves), 74 and 75 (halves, and whole ones), 0
@pytest.mark.parametrize("rows,K,N", [([128], 64, 1024), ([128, 0, 256, 128], 192, 3072), ([128] * 37, 128, 256), ([128] * 38, 64, 256), ([0, 0], 64, 256),
                                      ([256] * 9 + [128] * 2, 64, 1024), ([128] * 74, 64, 256), ([128] * 75, 64, 256),
                                      ([384, 128], 2112, 256), ([128] * 3, 448, 512)])  # fmt: skip
def test_split_tiles_give_the_same_sums(rows, K, N):
    cu, x, w, up, scale = _operands(rows, K, N, seed=K + N)
    n, status = int(cu[-1]), torch.zeros(8, dtype=torch.int32, device="cuda")
    for mode in ("plain", "swiglu", "scale"):
        kw = {"w_up": up} if mode == "swiglu" else {"row_scale": scale} if mode == "scale" else {}
        got = []
        for sms in (0, 2):  # two SMs: whole tiles
            pre = tuple(torch.full((x.shape[0], N), 5.0, device="cuda").bfloat16() for _ in range(2)) if mode == "swiglu" else None
            out = torch.full((x.shape[0], N), 3.0, device="cuda").bfloat16()
            grouped_gemm(x, w, cu, mode=mode, out=out, status=status, num_sms=sms, pair=False, save_pre=pre, **kw)
            got.append([out] + list(pre or ()))
        assert all(torch.equal(a, b) for a, b in zip(*got)), mode
        assert _close(got[0][0][:n], grouped_gemm_reference(x, w, cu, mode=mode, **kw)[:n]), mode
        assert bool((got[0][0][n:] == 3.0).all())
    assert int(status[0]) == 0
