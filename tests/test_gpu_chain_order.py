"""The state walks of packed batches in the order of their lengths, and of normalised dense rows in segments.
The order of the chains must not touch a bit: every sequence is compared with the same sequence run alone."""

import pytest
import torch

import kda_b200
from kda_b200 import _cabi
from oracle import kda_oracle as orc
from helpers import assert_normalised

pytestmark = pytest.mark.gpu


def _run(inp, spans=None, normalize=False, grad=True):
    leaves = [inp[n].bfloat16().cuda() for n in ("q", "k", "v")] + [inp["cum_gate"].cuda(), inp["beta"].cuda(),
                                                                   inp["h0"].cuda()]
    do = torch.randn(inp["v"].shape, generator=torch.Generator().manual_seed(61)).bfloat16().cuda()
    if spans is not None:
        a, b, i = spans
        leaves = [x[:, a:b].contiguous() for x in leaves[:5]] + [leaves[5][i:i + 1].contiguous()]
        do = do[:, a:b].contiguous()
    leaves = [x.requires_grad_(grad) for x in leaves]
    cu = None if spans is not None or inp["cu_seqlens"] is None else inp["cu_seqlens"].cuda()
    o, st = kda_b200.chunk_kda(*leaves, cu_seqlens=cu, output_final_state=True, normalize_qk=normalize)
    if not grad:
        return [o, st]
    return [o, st, *torch.autograd.grad([o, st], leaves, [do, 0.1 * torch.ones_like(st)])]


@pytest.mark.parametrize("sequences", [2, 5, 128, 129])      # 129: more than the kernels rank
def test_order_of_the_chains_does_not_touch_the_results(sequences):
    heads = 80 if sequences == 2 else (31 if sequences == 5 else 2)       # more chains than SMs
    lengths = [1 + (37 * i * i + 11 * i) % 331 for i in range(sequences)]
    lengths[-1] = 400                                        # the longest comes last
    if sequences > 2:
        lengths[1] = 0
        lengths[2] = lengths[-1]                             # a tie
    inp = orc.make_inputs(1, sum(lengths), heads, 128, 128, seed=62, with_state=True, lengths=lengths)
    whole = _run(inp)
    marks = inp["cu_seqlens"].tolist()
    for i in {0, 2 % sequences, sequences // 2, sequences - 1}:
        a, b = marks[i], marks[i + 1]
        if a == b:
            continue
        alone = _run(inp, (a, b, i))
        for n, (x, y) in enumerate(zip(whole, alone)):
            part = x[i:i + 1] if n in (1, 7) else x[:, a:b]
            assert torch.equal(part, y), (i, n)


@pytest.mark.parametrize("segments", [2, 3])
@pytest.mark.parametrize("gate_scale", [1.0, 0.02])
def test_normalised_rows_walked_in_segments(segments, gate_scale):
    inp = orc.make_inputs(2, 64 * 11 + 17, 2, 128, 128, seed=63, with_state=True)
    inp["cum_gate"] = inp["cum_gate"] * gate_scale
    serial = _run(inp, normalize=True)
    try:
        assert _cabi.lib().kda_set_row_segments(segments) == 0
        split = _run(inp, normalize=True)
        plain = _run(inp, normalize=True, grad=False)
    finally:
        _cabi.lib().kda_set_row_segments(0)
    # as for rows without the normalisation: the serial walk's bits almost everywhere when the gates forget,
    # else two bf16 evaluations of the boundary states
    for x, y in zip(split, serial):
        assert_normalised(x.float(), y.float(), 1e-4 if gate_scale == 1.0 else 1e-2, "segments")
    assert torch.equal(plain[0], split[0]) and torch.equal(plain[1], split[1])


@pytest.mark.parametrize("normalize", [False, True])
def test_kept_forward_of_a_long_row_and_its_gradients(normalize):
    """Two segments by the library's own choice (128 chunks, few chains): their states lie in the part of the kept
    buffer that the backward pass overwrites.  Against one segment per row, as above."""
    inp = orc.make_inputs(1, 64 * 128 + 17, 2, 128, 128, seed=64, with_state=True)
    split = _run(inp, normalize=normalize)
    try:
        assert _cabi.lib().kda_set_row_segments(1) == 0
        serial = _run(inp, normalize=normalize)
    finally:
        _cabi.lib().kda_set_row_segments(0)
    for x, y in zip(split, serial):
        assert_normalised(x.float(), y.float(), 1e-4, "segments")


@pytest.mark.parametrize("sequences,heads", [(2, 80), (5, 31), (17, 9), (128, 2)])
def test_long_chains_first_does_not_touch_the_results(sequences, heads):
    """Sequences long enough (4 + sequences / 8 chunks on average) for more chains than SMs to be ranked, with an empty
    one, a tie and the longest last."""
    mean = 64 * (4 + sequences // 8) + 40
    lengths = [1 + (37 * i * i + 11 * i) % (2 * mean) for i in range(sequences)]
    if sequences > 2:
        lengths[1], lengths[2] = 0, max(lengths)
    lengths[-1] = max(lengths) + (0 if sequences > 5 else mean)
    lengths[0] += max(0, mean * sequences - sum(lengths))
    gen = torch.Generator(device="cuda").manual_seed(65)
    r = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    tokens = sum(lengths)
    q, k = (torch.nn.functional.normalize(r(1, tokens, heads, 128), dim=-1).bfloat16() for _ in range(2))
    v, do = r(1, tokens, heads, 128).bfloat16(), r(1, tokens, heads, 128).bfloat16()
    gate, beta, h0 = -0.02 * torch.rand(1, tokens, heads, 128, generator=gen, device="cuda"), r(1, tokens, heads).sigmoid(), 0.02 * r(sequences, heads, 128, 128)
    marks = [0]
    for n in lengths:
        marks.append(marks[-1] + n)

    def run(args, cot, cu):
        leaves = [x.detach().contiguous().requires_grad_() for x in args]
        o, st = kda_b200.chunk_kda(*leaves, cu_seqlens=torch.tensor(cu, dtype=torch.int32, device="cuda"), output_final_state=True)
        return [o, st, *torch.autograd.grad([o, st], leaves, [cot, 0.1 * torch.ones_like(st)])]

    args = (q, k, v, gate, beta, h0)
    whole = run(args, do, marks)
    for i in sorted({0, 2 % sequences, sequences // 2, sequences - 1}):
        a, b = marks[i], marks[i + 1]
        if a == b:
            continue
        alone = run([x[:, a:b] for x in args[:5]] + [h0[i:i + 1]], do[:, a:b].contiguous(), [0, b - a])
        for n, (x, y) in enumerate(zip(whole, alone)):
            assert torch.equal(x[i:i + 1] if n in (1, 7) else x[:, a:b], y), (i, n)
