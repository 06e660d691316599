"""The sum of gradients in one pass: two to four of them and numbers it leaves to the general path, sizes around its blocks and
sizes it does not take; and the layer's input gradient through it."""

import pytest
import torch

import kda_b200

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [1, 2, 3, 4, 5])
@pytest.mark.parametrize("n", [0, 5, 8, 4096 - 8, 4096, 4096 + 8, 100000])
def test_sum_is_rounded_once(count, n):
    gen = torch.Generator(device="cuda").manual_seed(n)
    grads = [torch.randn(n, generator=gen, device="cuda").bfloat16() for _ in range(count)]
    want = grads[0].float()
    for t in grads[1:]:
        want = want + t.float()
    assert torch.equal(torch.ops.kda_b200_layer.sum_gradients(grads), want.bfloat16())
    torch.library.opcheck(torch.ops.kda_b200_layer.sum_gradients.default, (grads,), test_utils=("test_schema", "test_faketensor"))


class _OwnGate(kda_b200.KDAAttention):
    def gate_projections(self, hidden):
        return super().gate_projections(hidden)


@pytest.mark.parametrize("kind", [kda_b200.KDAAttention, _OwnGate])
def test_input_gradient(kind):
    """Against four passes that each reach the input through one projection only (their sums differ by roundings to bf16)."""
    torch.manual_seed(0)
    layer = kind(256, 2, 128, device="cuda")
    x = torch.randn(2, 70, 256, device="cuda").bfloat16().requires_grad_()
    d = torch.randn(2, 70, 256, device="cuda").bfloat16()
    (got,) = torch.autograd.grad([layer(x).hidden_states], [x], [d])
    parts = []
    for name in ("qkv_proj", "f_a_proj", "beta_proj", "g_a_proj"):
        one, linear = kda_b200.KDAAttention(256, 2, 128, device="cuda"), None
        one.load_state_dict(layer.state_dict())
        linear, wanted = one._linear, getattr(one, name)
        inputs = {id(getattr(one, n)) for n in ("qkv_proj", "f_a_proj", "beta_proj", "g_a_proj")}
        one._linear = lambda h, p: linear(h.detach() if id(p) in inputs and p is not wanted else h, p)
        (g,) = torch.autograd.grad([one(x).hidden_states], [x], [d])
        parts.append(g.double())
    want = sum(parts)
    # each part and the sum carry a rounding of 2^-9 relative to their own size
    assert ((got.double() - want).abs() <= 2.0 ** -8 * (want.abs() + sum(p.abs() for p in parts))).all()
