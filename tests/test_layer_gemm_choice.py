"""Which GEMMs of a layer run on CTA pairs, by the tiles of each product; what they give does not depend on it."""

import pytest
import torch

from moonep_b200 import Buffer
from moonep_b200.models.moe_layer import ExpertParallelMoE


def _layer(S, H, K, E, I):
    buf = Buffer(S, H, K, E, 1, num_sms=8, token_padding=128)
    return buf, ExpertParallelMoE(buf, I, init_std=0.05, seed=1)


@pytest.mark.gpu
def test_products_of_one_wave_of_pairs_take_single_ctas(monkeypatch):
    monkeypatch.delenv("MOONEP_GEMM_PAIR", raising=False)
    most = torch.cuda.get_device_properties(0).multi_processor_count // 2 // 8
    buf, layer = _layer(520, 256, 2, 4, 256)  # 260 rows per expert: two rows of tiles each
    assert [layer.forward_gemm_pair(n) for n in (0, 1, most, most + 1)] == [True, False, False, True]
    # a long contraction: half a wave; of one row of tiles each, from twice that length on
    assert [layer.forward_gemm_pair(n, d) for n, d in ((most, 2048), (most, 2112), (most // 2, 2112))] == [False, True, False]
    layer.destroy(), buf.destroy()
    buf, layer = _layer(512, 256, 2, 4, 256)
    assert [layer.forward_gemm_pair(2 * most, d) for d in (4096, 4160)] == [False, True]
    layer.destroy(), buf.destroy()
    buf, layer = _layer(256, 256, 2, 4, 256)  # 128 rows per expert
    assert not any(layer.forward_gemm_pair(n) for n in (0, 1, 1000))
    layer.destroy(), buf.destroy()


@pytest.mark.gpu
@pytest.mark.parametrize("S,H,K,E,I", [(520, 256, 2, 4, 256), (300, 512, 2, 3, 256), (1000, 256, 1, 2, 512)])
def test_pairs_and_single_ctas_give_the_same_step(S, H, K, E, I, monkeypatch):
    g = torch.Generator(device="cuda").manual_seed(S)
    x, dy = (torch.randn(S, H, generator=g, device="cuda").bfloat16() for _ in range(2))
    topk = torch.rand(S, E, generator=g, device="cuda").topk(K).indices.int()
    gates, tpe = torch.rand(S, K, generator=g, device="cuda"), torch.bincount(topk.flatten(), minlength=E).int()
    steps = []
    for switch in (None, "1"):
        if switch is None:
            monkeypatch.delenv("MOONEP_GEMM_PAIR", raising=False)
        else:
            monkeypatch.setenv("MOONEP_GEMM_PAIR", switch)
        buf, layer = _layer(S, H, K, E, I)
        out, saved = layer.forward(x, gates, topk, tpe)
        dx, dgates = layer.backward(saved, dy)
        layer.check()
        steps.append([t.clone() for t in (out, dx, dgates, *layer.owner_grads())])
        layer.destroy(), buf.destroy()
    for a, b in zip(*steps):  # bf16 roundings of the same fp32 sums: nothing, or a step apart where a sum's order differs
        assert float((a.float() - b.float()).abs().max()) <= 2.0**-7 * float(b.float().abs().max())
