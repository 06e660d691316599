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
