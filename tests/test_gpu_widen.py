"""The way of a weight gradient back to fp32: every 16-bit value exactly, sizes around the blocks of the kernel, sizes and
addresses it does not take, and the gradient of a layer's weights through it."""

import pytest
import torch

import kda_b200

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_every_value(dtype):
    x = torch.arange(65536, dtype=torch.int32).to(torch.int16).view(dtype).cuda()
    y = torch.ops.kda_b200_layer.widen(x)
    want = x.float()
    assert torch.equal(torch.isnan(y), torch.isnan(want))
    assert torch.equal(y.nan_to_num(0.0), want.nan_to_num(0.0))


@pytest.mark.parametrize("n", [0, 1, 4, 8, 2048 * 4 - 8, 2048 * 4, 2048 * 4 + 8, 100003])
@pytest.mark.parametrize("offset", [0, 1])
def test_sizes_and_addresses(n, offset):
    x = torch.randn(n + offset, device="cuda").bfloat16()[offset:]
    assert torch.equal(torch.ops.kda_b200_layer.widen(x), x.float())
    t = torch.randn(24, 40, device="cuda").bfloat16().t()
    assert torch.equal(torch.ops.kda_b200_layer.widen(t), t.float())
    torch.library.opcheck(torch.ops.kda_b200_layer.widen.default, (t,), test_utils=("test_schema", "test_faketensor"))


@pytest.mark.parametrize("hidden,heads,large", [(256, 2, False), (2048, 32, True), (2040, 32, False)])
def test_layer_weight_gradients_are_those_of_a_plain_cast(hidden, heads, large):
    """Either side of the size from which a weight has its own way back."""
    torch.manual_seed(0)
    layer = kda_b200.KDAAttention(hidden, heads, 128, device="cuda")
    x = torch.randn(2, 70, hidden, device="cuda").bfloat16()
    w = layer.out_proj.weight
    d = torch.randn(2, 70, hidden, device="cuda").bfloat16()
    assert (type(layer._cast(layer.out_proj).grad_fn).__name__ == "_CastWeightBackward") == large
    seen = {}
    hook = layer.out_proj.weight.register_hook(lambda g: seen.setdefault("grad", g))
    inner = {}
    linear = torch.nn.functional.linear

    def recording(a, weight, *rest):
        if weight.shape == w.shape and a.shape[-1] == w.shape[1]:
            inner["a"] = a.detach()
        return linear(a, weight, *rest)

    torch.nn.functional.linear = recording
    try:
        out = layer(x).hidden_states
    finally:
        torch.nn.functional.linear = linear
    out.backward(d)
    hook.remove()
    plain = w.detach().clone().requires_grad_()
    torch.nn.functional.linear(inner["a"], plain.to(torch.bfloat16)).backward(d)
    assert seen["grad"].dtype == torch.float32 and torch.equal(seen["grad"], plain.grad)
