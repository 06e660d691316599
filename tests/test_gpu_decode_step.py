"""decode_step (one call, two overlapping launches) against its two operators run one after the other: the same
kernels, so the same bits.  Many steps without a synchronisation, because the state update of a step starts
before its preprocessing has finished and after the step before it."""

import pytest
import torch

import kda_b200

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sequences,heads,width,dtype", [
    (1, 1, 4, torch.bfloat16),
    (1, 32, 4, torch.bfloat16),
    (5, 3, 2, torch.float16),
    (37, 32, 4, torch.bfloat16),
    (7, 2, 5, torch.float32),            # the scalar preprocessing kernel
    (300, 32, 4, torch.bfloat16),        # several preprocessing waves, 65 states per block
])
def test_equals_its_two_operators_over_many_steps(sequences, heads, width, dtype):
    gen = torch.Generator(device="cuda").manual_seed(51)
    r = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    channels, slots, steps = 3 * heads * 128, sequences + 2, 12
    weight = (0.5 * r(channels, width)).to(dtype)
    conv_a = r(slots, width - 1, channels).to(dtype)
    pool_a = 0.02 * r(slots, heads, 128, 128)
    conv_b, pool_b = conv_a.clone(), pool_a.clone()
    a_log, bias = 0.1 * r(heads), 0.1 * r(heads, 128)
    idx = torch.randperm(slots - 1, generator=gen, device="cuda").int()[:sequences] + 1
    if sequences > 2:
        idx[1] = 0                       # a padding row
    xs = [r(sequences, channels).to(dtype) for _ in range(steps)]
    raws = [r(sequences, heads, 128).to(dtype) for _ in range(steps)]
    betas = [r(sequences, heads).sigmoid() for _ in range(steps)]
    with torch.no_grad():
        got = [kda_b200.decode_step(x, weight, conv_a, g, a_log, bias, b, pool_a, idx)
               for x, g, b in zip(xs, raws, betas)]
        want = []
        for x, g, b in zip(xs, raws, betas):
            q, k, v, gate = torch.ops.kda_b200.kda_decode_prep(x, weight, conv_b, idx, g, a_log, bias, heads,
                                                               "silu", -5.0, 1e-6)
            torch.cuda.synchronize()
            o, _ = kda_b200.recurrent_kda(q, k, v, gate, b.reshape(sequences, 1, heads), pool_b, state_indices=idx)
            torch.cuda.synchronize()
            want.append(o.reshape(sequences, heads, 128))
    for a, b in zip(got, want):
        assert torch.equal(a, b)
    assert torch.equal(pool_a, pool_b) and torch.equal(conv_a, conv_b)


def test_rejections_are_those_of_the_two_operators():
    gen = torch.Generator(device="cuda").manual_seed(52)
    r = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    x, w, conv = r(2, 384), r(384, 4), r(3, 3, 384)
    raw, a_log, bias, beta, pool = r(2, 1, 128), r(1), r(1, 128), r(2, 1), r(3, 1, 128, 128)
    idx = torch.tensor([1, 2], dtype=torch.int32, device="cuda")
    step = lambda **kw: kda_b200.decode_step(**{**dict(x=x, conv_weight=w, conv_state=conv, raw_gate=raw, A_log=a_log,
                                                       dt_bias=bias, beta=beta, state_pool=pool, state_indices=idx), **kw})
    with pytest.raises(ValueError):
        step(x=x[:0], raw_gate=raw[:0], beta=beta[:0], state_indices=idx[:0])
    with pytest.raises(TypeError):
        step(beta=beta.double())
    with pytest.raises(ValueError):
        step(beta=beta.cpu())
    with pytest.raises(RuntimeError):
        step(state_pool=pool.clone().requires_grad_())
