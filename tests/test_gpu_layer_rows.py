"""A layer whose own convolution returns rows of another dtype than bf16 runs as before."""

import pytest
import torch

import kda_b200

pytestmark = pytest.mark.gpu


class _OwnConvolution(kda_b200.KDAAttention):
    """A convolution that returns its rows in another dtype."""

    rows = torch.float32

    def short_convolution(self, qkv, initial_state, **options):
        out, final = super().short_convolution(qkv, initial_state, **options)
        return out.to(self.rows), final


@pytest.mark.parametrize("rows", [torch.float32, torch.float16])
@pytest.mark.parametrize("packed", [False, True])
def test_a_convolution_that_returns_other_rows(rows, packed):
    torch.manual_seed(0)
    plain = kda_b200.KDAAttention(256, 2, 128, device="cuda")
    own = _OwnConvolution(256, 2, 128, device="cuda")
    own.rows = rows
    own.load_state_dict(plain.state_dict())
    x = torch.randn(1, 150, 256, device="cuda").bfloat16()
    cu = torch.tensor([0, 65, 150], dtype=torch.int32, device="cuda") if packed else None
    results = []
    for layer in (plain, own):
        leaf = x.clone().requires_grad_()
        out = layer(leaf, cu_seqlens=cu, return_final_state=True)
        out.hidden_states.float().square().sum().backward()
        results.append((out.hidden_states, out.final_state, leaf.grad))
    for got, want in zip(results[1], results[0]):
        # the rows go back to bf16 for the core (exactly, or by one more rounding from fp16); what is left are roundings behind it
        assert float((got.double() - want.double()).norm() / want.double().norm()) < 2.0 ** -6
