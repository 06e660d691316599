"""The three narrow projections of the layer in one GEMM against the same layer with its projections apart: outputs and all
gradients, dense, packed with an unused tail, and without gradients; widths that stay apart."""

import pytest
import torch

import kda_b200

pytestmark = pytest.mark.gpu


class _Apart(kda_b200.KDAAttention):
    def gate_projections(self, hidden):
        return super().gate_projections(hidden)


def _pair(heads, hidden, **kw):
    torch.manual_seed(heads)
    joint = kda_b200.KDAAttention(hidden, heads, 128, device="cuda", **kw)
    apart = _Apart(hidden, heads, 128, device="cuda", **kw)
    apart.load_state_dict(joint.state_dict())
    return joint, apart


def _close(got, want, what):
    # bf16 values on both sides, from GEMMs that sum in another order: a few roundings of 2^-9 carried through the layer
    err = float((got.double() - want.double()).norm() / want.double().norm().clamp_min(1e-30))
    assert err < 2.0 ** -6, (what, err)


@pytest.mark.parametrize("heads,joined", [(8, True), (16, True), (3, False)])
@pytest.mark.parametrize("packed", [False, True])
def test_joint_projections(heads, joined, packed):
    joint, apart = _pair(heads, 256, mask_inactive_capacity=packed)
    batch, tokens, used = (1, 200, 187) if packed else (2, 70, 70)
    cu = torch.tensor([0, 65, 65, 187], dtype=torch.int32, device="cuda") if packed else None
    x = torch.randn(batch, tokens, 256, device="cuda").bfloat16()
    if packed:
        x[:, used:] = float("nan")
    d = torch.randn(batch, tokens, 256, device="cuda").bfloat16()
    assert (joint._narrow_projections(x) is not None) == joined and apart._narrow_projections(x) is None
    results = []
    for layer in (joint, apart):
        leaf = x.clone().requires_grad_()
        out = layer(leaf, cu_seqlens=cu).hidden_states
        out[:, :used].backward(d[:, :used])
        results.append((out[:, :used].detach(), leaf.grad[:, :used], {n: p.grad for n, p in layer.named_parameters()}))
    _close(results[0][0], results[1][0], "output")
    _close(results[0][1], results[1][1], "input gradient")
    for name, want in results[1][2].items():
        got = results[0][2][name]
        assert got.dtype == torch.float32 and torch.isfinite(got).all()
        _close(got, want, name)
    with torch.no_grad():
        again = joint(x, cu_seqlens=cu).hidden_states[:, :used]
    assert torch.equal(again, results[0][0])


def test_only_some_weights_train():
    joint, apart = _pair(8, 256)
    x, d = (torch.randn(1, 64, 256, device="cuda").bfloat16() for _ in range(2))
    for layer in (joint, apart):
        for p in (layer.f_a_proj, layer.beta_proj):
            p.weight.requires_grad_(False)
        layer(x).hidden_states.backward(d)
        assert layer.f_a_proj.weight.grad is None and layer.beta_proj.weight.grad is None
    _close(joint.g_a_proj.weight.grad, apart.g_a_proj.weight.grad, "g_a_proj")


class _OwnLinear(kda_b200.KDAAttention):
    def _linear(self, x, layer):
        self.seen = getattr(self, "seen", []) + [layer]
        return super()._linear(x, layer)


def test_a_replaced_linear_sees_every_projection():
    torch.manual_seed(1)
    plain = kda_b200.KDAAttention(256, 8, 128, device="cuda")
    own = _OwnLinear(256, 8, 128, device="cuda")
    own.load_state_dict(plain.state_dict())
    x = torch.randn(2, 70, 256, device="cuda").bfloat16()
    _close(own(x).hidden_states, plain(x).hidden_states, "output")
    want = {own.qkv_proj, own.f_a_proj, own.f_b_proj, own.beta_proj, own.g_a_proj, own.g_b_proj, own.out_proj}
    assert set(own.seen) == want and len(own.seen) == len(want)
    plain._linear = lambda inputs, layer: _OwnLinear._linear(own, inputs, layer)         # replaced on the object
    assert plain._narrow_projections(x) is None


class _Marked(torch.Tensor):
    pass


def test_weights_of_another_tensor_class_stay_apart():
    layer = kda_b200.KDAAttention(256, 8, 128, device="cuda")
    x = torch.randn(1, 8, 256, device="cuda").bfloat16()
    assert layer._narrow_projections(x) is not None
    layer.f_a_proj.weight = torch.nn.Parameter(layer.f_a_proj.weight.detach().as_subclass(_Marked))
    assert layer._narrow_projections(x) is None
