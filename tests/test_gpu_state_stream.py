"""One token per sequence by state streaming, where its ring, its operand slots and its grid end: one state, as many states
as SMs and one more, several turns of the three stages and eight slots, padding first, last and in between, slots that only
one of the two pools has, operands of every dtype and alignment; against the fp64 recurrence."""

import pytest
import torch

import kda_b200
from oracle import kda_oracle as orc

pytestmark = pytest.mark.gpu

# fp32 sums of 128 terms and one update: 128 * 2^-24 = 8e-6 of the largest value; outputs of 16-bit rows one rounding more
TOL = {torch.float32: 1e-5, torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11 + 1e-5}


def _err(a, b):
    return float((a.double().cpu() - b).abs().max() / b.abs().max())


@pytest.mark.parametrize("seqs,heads,dtype,offset", [
    (1, 1, torch.float32, 0), (1, 3, torch.bfloat16, 0), (37, 4, torch.float16, 1), (149, 1, torch.bfloat16, 1),
    (74, 32, torch.bfloat16, 0), (25, 32, torch.float32, 1),
])
@pytest.mark.parametrize("paged", [False, True])
def test_one_token_per_sequence(seqs, heads, dtype, offset, paged):
    gen = torch.Generator().manual_seed(seqs + heads)
    r = lambda *s: torch.randn(*s, generator=gen)

    def place(x):          # on the GPU, `offset` elements past an aligned address
        flat = torch.empty(x.numel() + offset, dtype=x.dtype, device="cuda")
        flat[offset:].copy_(x.reshape(-1))
        return flat[offset:].view(x.shape)

    q, k = (torch.nn.functional.normalize(r(seqs, 1, heads, 128), dim=-1).to(dtype) for _ in range(2))
    v, g, beta = r(seqs, 1, heads, 128).to(dtype), -torch.rand(seqs, 1, heads, 128, generator=gen), r(seqs, 1, heads).sigmoid()
    h0 = r(seqs, heads, 128, 128)
    want_o, want_s = orc.recurrent_kda_ref(*(x.double() for x in (q, k, v, g, beta, h0)))
    args = [place(x) for x in (q, k, v, g, beta)]
    if not paged:
        o, s = kda_b200.recurrent_kda(*args, h0.cuda(), output_final_state=True)
    else:
        slots = torch.randperm(seqs, generator=gen).int() + 1
        pads = sorted({0, seqs // 2, seqs - 1}) if seqs > 1 else []
        pool = torch.full((seqs + 1, heads, 128, 128), 7.0)
        pool[slots.long()] = h0
        slots[pads] = torch.tensor([0, -1, seqs + 1], dtype=torch.int32)[:len(pads)]
        before = pool.clone()
        pool = pool.cuda()
        o, _ = kda_b200.recurrent_kda(*args, pool, state_indices=slots.cuda())
        s = pool.cpu()
        kept = torch.ones(seqs + 1, dtype=torch.bool)
        live = slots.clone()
        live[pads] = 0
        kept[live[live > 0].long()] = False
        assert torch.equal(s[kept], before[kept])
        rows = [i for i in range(seqs) if i not in pads]
        s, want_s = s[slots[rows].long()], want_s[rows]
        want_o[pads] = 0
        assert not o[pads].any()
    assert _err(o, want_o) < TOL[dtype]
    assert _err(s, want_s) < 1e-5


def test_slots_that_only_one_pool_has():
    """A history slot beyond the state pool advances the history alone; a state slot beyond the history pool sees zero
    operands and a unit decay: what preprocessing and state update do one after the other."""
    gen = torch.Generator(device="cuda").manual_seed(3)
    r = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    heads, bf16 = 2, torch.bfloat16
    for conv_slots, state_slots in ((4, 2), (2, 4)):
        x, w, raw = r(2, 768).to(bf16), r(768, 4).to(bf16), r(2, heads, 128).to(bf16)
        conv, pool = r(conv_slots, 3, 768).to(bf16), r(state_slots, heads, 128, 128)
        a_log, bias, beta = r(heads), r(heads, 128), r(2, heads).sigmoid()
        idx = torch.tensor([1, 3], dtype=torch.int32, device="cuda")
        conv2, pool2 = conv.clone(), pool.clone()
        with torch.no_grad():
            out = kda_b200.decode_step(x, w, conv, raw, a_log, bias, beta, pool, idx)
            q, k, v, g = torch.ops.kda_b200.kda_decode_prep(x, w, conv2, idx, raw, a_log, bias, heads, "silu", -5.0, 1e-6)
            o, _ = kda_b200.recurrent_kda(q, k, v, g, beta.view(2, 1, heads), pool2, state_indices=idx)
        assert torch.equal(out, o.view(2, heads, 128))
        assert torch.equal(conv, conv2) and torch.equal(pool, pool2)
