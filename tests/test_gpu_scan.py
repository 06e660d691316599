"""The token scan at the edges of its tiles: head sizes around the row groups (32, 64, 128, 256), value
columns that end inside a CTA's slice, token counts around the operand tiles (4, 8, 16), and both column
layouts (few chains / many chains), against the fp64 recurrence."""

import pytest
import torch

import kda_b200
from oracle import kda_oracle as orc

pytestmark = pytest.mark.gpu

# fp32 products and sums of at most 256 terms, carried over at most 33 tokens of a contracting
# recurrence: 33 * 256 * 2^-24 = 5e-4 of the largest value bounds the worst case
TOL = 5e-4


def _close(got, want, what):
    err = float((got.double().cpu() - want).abs().max() / want.abs().max().clamp_min(1e-30))
    assert err < TOL, (what, err)


@pytest.mark.parametrize("heads", [2, 80], ids=["few-chains", "many-chains"])
@pytest.mark.parametrize("kd,vd", [(32, 32), (33, 20), (64, 68), (96, 128), (128, 132), (129, 16), (256, 36)])
def test_scan_tile_edges(heads, kd, vd):
    lengths = [1, 0, 3, 4, 5, 7, 8, 9, 15, 16, 17, 33]
    inp = orc.make_inputs(1, sum(lengths), heads, kd, vd, seed=kd + vd, with_state=True, lengths=lengths)
    dev = {n: t.cuda() if torch.is_tensor(t) else t for n, t in inp.items()}
    want_o, want_s = orc.recurrent_kda_ref(*(inp[n].double() for n in ("q", "k", "v", "gate_log2", "beta", "h0")),
                                           inp["cu_seqlens"])
    args = (dev["q"], dev["k"], dev["v"])
    o, s = kda_b200.recurrent_kda(*args, dev["gate_log2"], dev["beta"], dev["h0"],
                                  cu_seqlens=dev["cu_seqlens"], output_final_state=True)
    _close(o, want_o, "output")
    _close(s, want_s, "state")
    # the same from the cumulative gate of chunk_kda: the difference of two prefix sums of up to 64 gates
    # (at most 2^9) adds 2^9 * 2^-24 * ln 2 to the relative error of a decay
    o, s = kda_b200.chunk_kda(*args, dev["cum_gate"], dev["beta"], dev["h0"], cu_seqlens=dev["cu_seqlens"],
                              output_final_state=True, exact_fp32=True)
    _close(o, want_o, "output (cumulative gate)")
    _close(s, want_s, "state (cumulative gate)")


def test_cumulative_gate_restarts_at_every_chunk_and_row():
    inp = orc.make_inputs(2, 131, 3, 40, 24, seed=4, with_state=True)
    dev = {n: t.cuda() if torch.is_tensor(t) else t for n, t in inp.items()}
    want_o, want_s = orc.recurrent_kda_ref(*(inp[n].double() for n in ("q", "k", "v", "gate_log2", "beta", "h0")))
    o, s = kda_b200.chunk_kda(dev["q"], dev["k"], dev["v"], dev["cum_gate"], dev["beta"], dev["h0"],
                              output_final_state=True)
    _close(o, want_o, "output")
    _close(s, want_s, "state")
    torch.library.opcheck(torch.ops.kda_b200_fused.chunk_scan.default,
                          (dev["q"], dev["k"], dev["v"], dev["cum_gate"], dev["beta"], dev["h0"], None, True),
                          test_utils=("test_schema", "test_faketensor"))


FORMS = [  # kd, vd, heads, lengths: what the average length and the number of 16-column slices select
    (33, 20, 2, [1, 1, 1]), (64, 33, 3, [1] * 5), (128, 130, 2, [1, 1]), (20, 5, 1, [1, 1]),                # short, one token
    (129, 16, 2, [1, 1]), (256, 36, 3, [1, 3, 0, 1, 0]), (64, 64, 3, [0, 1, 2, 1]),
    (64, 64, 12, [3, 1, 5, 0, 1]), (96, 50, 12, [2] * 5), (192, 64, 24, [2, 0, 3, 3, 1]),                 # short, two tokens
    (128, 130, 12, [9, 0, 1, 17, 8]), (64, 33, 40, [3, 2, 16, 0]), (32, 30, 50, [2, 2, 33, 1]),           # 32 columns per CTA
    (100, 65, 16, [1, 1, 64, 65]), (128, 64, 12, [3, 5, 4, 0, 6]), (96, 96, 16, [6, 4]),                  # wide from one turn on
]


@pytest.mark.parametrize("kd,vd,heads,lengths", FORMS)
@pytest.mark.parametrize("paged", [False, True])
def test_every_form_of_the_scan(kd, vd, heads, lengths, paged):
    inp = orc.make_inputs(1, sum(lengths) + 1, heads, kd, vd, seed=kd + vd, with_state=True, lengths=lengths)
    dev = {n: t.cuda() if torch.is_tensor(t) else t for n, t in inp.items()}
    want_o, want_s = orc.recurrent_kda_ref(*(inp[n].double() for n in ("q", "k", "v", "gate_log2", "beta", "h0")),
                                           inp["cu_seqlens"])
    args = (dev["q"], dev["k"], dev["v"], dev["gate_log2"], dev["beta"])
    n = len(lengths)
    if not paged:
        o, s = kda_b200.chunk_kda(*args[:3], dev["cum_gate"], dev["beta"], dev["h0"], cu_seqlens=dev["cu_seqlens"],
                                  output_final_state=True, exact_fp32=True)        # the same from the cumulative gate
        _close(o, want_o, "output (cumulative gate)")
        _close(s, want_s, "state (cumulative gate)")
        o, s = kda_b200.recurrent_kda(*args, dev["h0"], cu_seqlens=dev["cu_seqlens"], output_final_state=True)
    else:                                       # slots in reverse order behind an unused one; the last sequence is padding
        slots = torch.arange(n, 0, -1, dtype=torch.int32)
        slots[-1] = 0
        pool = torch.full((n + 1, heads, kd, vd), 7.0)
        pool[slots[:-1].long()] = inp["h0"][:-1]
        pool = pool.cuda()
        o, _ = kda_b200.recurrent_kda(*args, pool, cu_seqlens=dev["cu_seqlens"], state_indices=slots.cuda())
        marks = inp["cu_seqlens"].tolist()
        want_o[:, marks[-2]:] = 0
        want_s[-1] = 7.0
        assert torch.equal(pool[0].cpu(), torch.full_like(pool[0].cpu(), 7.0))
        s = pool[torch.arange(n, 0, -1)]        # (slot 1 belongs to nobody and keeps its sevens)
    _close(o, want_o, "output")
    _close(s, want_s, "state")
