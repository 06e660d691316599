"""KDAAttention traced as one graph, forward and backward, with the bits of the eager call: small weights that are cast by ``.to``,
weights that have their own way back to fp32, and the narrow projections apart or in one GEMM."""

import pytest
import torch

import kda_b200

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("hidden,heads", [(256, 2), (2048, 33), (256, 8), (2048, 32)])
def test_one_graph(hidden, heads):
    torch.manual_seed(heads)
    layer = kda_b200.KDAAttention(hidden, heads, 128, device="cuda")
    x, d = (torch.randn(2, 70, hidden, device="cuda").bfloat16() for _ in range(2))

    def step(call):
        leaf = x.clone().requires_grad_()
        out = call(leaf).hidden_states
        return [out, *torch.autograd.grad(out, [leaf, *layer.parameters()], d)]

    torch._dynamo.reset()
    for got, want in zip(step(torch.compile(layer, fullgraph=True, backend="aot_eager")), step(layer)):
        assert torch.equal(got, want)
