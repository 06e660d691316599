"""Contiguous inputs off the addresses that a kernel's vector loads need: refused on the host, or taken by another form, and never handed
to the vector loads (a misaligned one takes the CUDA context down)."""

import pytest
import torch

import kda_b200
from kda_b200 import _cabi

pytestmark = pytest.mark.gpu


def _off(x, elements=1):
    flat = torch.empty(x.numel() + elements, dtype=x.dtype, device=x.device)
    flat[elements:].copy_(x.reshape(-1))
    return flat[elements:].view(x.shape)


def _core(tokens=130, batch=1):
    gen = torch.Generator(device="cuda").manual_seed(tokens)
    r = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    q, k, v = (torch.nn.functional.normalize(r(batch, tokens, 2, 128), dim=-1).bfloat16() for _ in range(3))
    gate = -0.01 * torch.rand(batch, tokens, 2, 128, generator=gen, device="cuda")
    return q, k, v, gate, r(batch, tokens, 2).sigmoid(), 0.1 * r(batch, 2, 128, 128)


def _refused(call):
    with pytest.raises(RuntimeError, match="invalid argument"):
        call()
    torch.cuda.synchronize()


def test_states_of_the_chunked_core():
    q, k, v, gate, beta, h0 = _core()
    for extra in ({}, {"normalize_qk": True}):
        _refused(lambda: kda_b200.chunk_kda(q, k, v, gate, beta, _off(h0), output_final_state=True, **extra))
    leaves = [x.clone().requires_grad_() for x in (q, k, v, gate, beta, h0)]
    for recompute in (False, True):
        o, s = kda_b200.chunk_kda(*leaves, output_final_state=True, recompute=recompute)
        _refused(lambda: torch.autograd.grad([o, s], leaves, [torch.ones_like(o), _off(torch.ones_like(s))]))
    # rows walked in segments read it element by element
    try:
        assert _cabi.lib().kda_set_row_segments(2) == 0
        args = _core(64 * 8)
        want = kda_b200.chunk_kda(*args, output_final_state=True)
        got = kda_b200.chunk_kda(*args[:5], _off(args[5]), output_final_state=True)
    finally:
        _cabi.lib().kda_set_row_segments(0)
    assert all(torch.equal(a, b) for a, b in zip(got, want))


def test_gate():
    raw, a, b = torch.randn(1, 70, 2, 128, device="cuda").bfloat16(), torch.zeros(2, device="cuda"), torch.zeros(2, 128, device="cuda")
    want = kda_b200.bounded_gate_cumsum(raw, a, b)
    _refused(lambda: kda_b200.bounded_gate_cumsum(_off(raw), a, b))
    _refused(lambda: kda_b200.bounded_gate_cumsum(raw, a, _off(b)))
    assert torch.equal(kda_b200.bounded_gate_cumsum(_off(raw, 4), _off(a), b), want)            # four elements are enough
    leaf = raw.clone().requires_grad_()
    _refused(lambda: torch.autograd.grad(kda_b200.bounded_gate_cumsum(leaf, a, b), [leaf], [_off(torch.ones_like(want))]))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
@pytest.mark.parametrize("width", [3, 4])
def test_convolution(dtype, width):
    x, w, h = (torch.randn(*s, device="cuda").to(dtype) for s in ((1, 70, 16), (16, width), (1, width - 1, 16)))
    want = kda_b200.causal_conv1d(x, w, initial_state=h)
    _refused(lambda: kda_b200.causal_conv1d(_off(x), w, initial_state=h))
    _refused(lambda: kda_b200.causal_conv1d(x, w, initial_state=_off(h)))
    if width == 4:
        _refused(lambda: kda_b200.causal_conv1d(x, _off(w), initial_state=h))
    assert torch.equal(kda_b200.causal_conv1d(x, _off(w, 4), initial_state=h), want)
    leaf = x.clone().requires_grad_()
    _refused(lambda: torch.autograd.grad(kda_b200.causal_conv1d(leaf, w), [leaf], [_off(torch.ones_like(want))]))
    state = torch.zeros(3, width - 1, 16, device="cuda", dtype=dtype)
    _refused(lambda: kda_b200.causal_conv1d_decode(_off(x[0, :2].contiguous()), w, state))
    _refused(lambda: kda_b200.causal_conv1d_decode(x[0, :2], w, _off(state)))


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_l2norm_and_output_gate(dtype):
    x = torch.randn(9, 128, device="cuda").to(dtype)
    _refused(lambda: kda_b200.l2norm(_off(x)))
    torch.testing.assert_close(kda_b200.l2norm(_off(x, 4)), kda_b200.l2norm(x))
    weight = torch.ones(128, device="cuda")
    torch.testing.assert_close(kda_b200.gated_output_norm(_off(x), _off(x), _off(weight)),
                               kda_b200.gated_output_norm(x, x, weight))
