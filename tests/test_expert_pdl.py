"""Expert kernels launched behind one another (programmatic dependent launch) give what they give in stream order."""

import pytest
import torch

from moonep_b200 import Buffer
from moonep_b200.models.moe_layer import ExpertParallelMoE
from moonep_b200.models.routing import make_routing

pytestmark = pytest.mark.gpu


# rows per expert below and above 128 (one CTA per tile, CTA pairs), groups with odd and even numbers of row blocks
@pytest.mark.parametrize("S,K,E", [(24, 2, 4), (700, 3, 5)])
def test_layer_steps_with_and_without(S, K, E, monkeypatch):
    H, I = 256, 256

    def steps(pdl):
        monkeypatch.setenv("MOONEP_PDL", pdl)
        buf = Buffer(S, H, K, E, 1, num_sms=8, token_padding=128)
        layer = ExpertParallelMoE(buf, I, init_std=0.05, seed=3)
        out = []
        for step in range(6):  # buffers of one step are the next one's: an early reader or writer would show
            g = torch.Generator().manual_seed(step)
            x = torch.randn(S, H, generator=g).to(torch.bfloat16).cuda()
            go = torch.randn(S, H, generator=g).to(torch.bfloat16).cuda()
            topk, tpe, gates = make_routing("softmax", S, K, E, 1, 0, seed=step)
            y, saved = layer.forward(x, gates.cuda(), topk.cuda(), tpe.cuda())
            dx, dg = layer.backward(saved, go)
            layer.sgd_step(1e-3)
            layer.zero_grad()
            out += [y, dx, dg]
        layer.check()
        out += [w.clone() for w in layer.owner_weights()] + [t.clone() for t in layer.owner_grads()]
        layer.destroy()
        buf.destroy()
        return out

    for a, b in zip(steps("1"), steps("0")):
        assert torch.equal(a, b)


@pytest.mark.parametrize("S,K,E", [(24, 2, 4), (700, 3, 5)])
def test_captured_forward_follows_its_inputs(S, K, E):
    """The same kernels as nodes of a graph: replays on new inputs equal the calls."""
    buf = Buffer(S, 256, K, E, 1, num_sms=8, token_padding=128)
    layer = ExpertParallelMoE(buf, 256, init_std=0.05, seed=3)
    g = torch.Generator().manual_seed(1)
    x = torch.randn(S, 256, generator=g).to(torch.bfloat16).cuda()
    topk, tpe, gates = (t.cuda() for t in make_routing("softmax", S, K, E, 1, 0, seed=1))
    step = buf.capture(lambda: layer.forward(x, gates, topk, tpe, save_for_backward=False)[0])
    for i in range(3):
        new = make_routing("softmax", S, K, E, 1, 0, seed=10 + i)
        for dst, src in zip((topk, tpe, gates), new):
            dst.copy_(src)
        x.copy_(torch.randn(S, 256, generator=g))
        got = step.replay().clone()
        want = layer.forward(x, gates, topk, tpe, save_for_backward=False)[0]
        assert torch.equal(got, want)
    layer.check()
    layer.destroy()
    buf.destroy()
