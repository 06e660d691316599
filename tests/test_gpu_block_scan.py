"""The scan in blocks of four tokens (fp32 operands) where its blocks, tiles and moving warps end: token counts around 4, 8, 16 and 32,
head sizes around its row groups (32, 64, 128) and column slices (16), chunk boundaries of the cumulative gate, gates that forget at
once; the wide forms with each number of columns per block; against the fp64 recurrence."""

import pytest
import torch

import kda_b200
from oracle import kda_oracle as orc

pytestmark = pytest.mark.gpu

# fp32 sums of at most 128 terms over at most 200 tokens of a contracting recurrence, whose roundings of 2^-24 have either sign:
# sqrt(200 * 128) * 2^-24 = 1e-5 of the largest value
TOL = 1e-5


def _close(got, want, what):
    err = float((got.double().cpu() - want).abs().max() / want.abs().max().clamp_min(1e-30))
    assert err < TOL, (what, err)


@pytest.mark.parametrize("kd,vd", [(20, 5), (32, 16), (33, 17), (64, 64), (96, 33), (128, 128)])
@pytest.mark.parametrize("lengths", [[5, 0, 7, 12, 31, 1], [15, 16, 17, 32, 33], [64, 65, 200]], ids=str)
def test_block_and_tile_edges(kd, vd, lengths):
    inp = orc.make_inputs(1, sum(lengths), 2, kd, vd, seed=kd + len(lengths), with_state=True, lengths=lengths)
    dev = {n: t.cuda() if torch.is_tensor(t) else t for n, t in inp.items()}
    want_o, want_s = orc.recurrent_kda_ref(*(inp[n].double() for n in ("q", "k", "v", "gate_log2", "beta", "h0")),
                                           inp["cu_seqlens"])
    args = (dev["q"], dev["k"], dev["v"])
    o, s = kda_b200.recurrent_kda(*args, dev["gate_log2"], dev["beta"], dev["h0"], cu_seqlens=dev["cu_seqlens"],
                                  output_final_state=True)
    _close(o, want_o, "output")
    _close(s, want_s, "state")
    o, s = kda_b200.chunk_kda(*args, dev["cum_gate"], dev["beta"], dev["h0"], cu_seqlens=dev["cu_seqlens"],
                              output_final_state=True, exact_fp32=True)
    _close(o, want_o, "output (cumulative gate)")
    _close(s, want_s, "state (cumulative gate)")


def test_mixed_dtypes_and_gates_that_forget():
    inp = orc.make_inputs(2, 37, 3, 64, 40, seed=9, with_state=True)
    q, k, v = inp["q"].bfloat16(), inp["k"].half(), inp["v"].bfloat16()
    gate = inp["gate_log2"].clone()
    gate[:, 5] = -300.0                    # 2^g is zero in fp32
    gate[:, 18, :, ::2] = float("-inf")
    want_o, want_s = orc.recurrent_kda_ref(q.double(), k.double(), v.double(), gate.double(), inp["beta"].double(),
                                           inp["h0"].double())
    o, s = kda_b200.recurrent_kda(q.cuda(), k.cuda(), v.cuda(), gate.cuda(), inp["beta"].cuda(), inp["h0"].cuda(),
                                  output_final_state=True)
    assert torch.isfinite(o.float()).all() and torch.isfinite(s).all()
    err = float((o.double().cpu() - want_o).abs().max() / want_o.abs().max())
    assert err < 2.0 ** -8 + TOL
    _close(s, want_s, "state")


@pytest.mark.parametrize("dtypes", ["mixed", "fp32"])
def test_forgetting_in_every_form(dtypes):
    """Decays of zero inside a block of fp32 operands, and token by token for the others."""
    inp = orc.make_inputs(1, 45, 2, 48, 24, seed=4, with_state=True)
    if dtypes == "mixed":
        inp["k"] = inp["k"].bfloat16()
    inp["gate_log2"][:, 6] = -300.0
    inp["gate_log2"][:, 11:13] = float("-inf")
    args = [inp[n] for n in ("q", "k", "v", "gate_log2", "beta", "h0")]
    want_o, want_s = orc.recurrent_kda_ref(*(x.double() for x in args))
    o, s = kda_b200.recurrent_kda(*(x.cuda() for x in args), output_final_state=True)
    _close(o, want_o, "output")
    _close(s, want_s, "state")


@pytest.mark.parametrize("kd,vd", [(32, 40), (32, 64), (20, 100), (32, 128), (17, 196)])
@pytest.mark.parametrize("heads,lengths", [(8, [4, 1, 0, 3, 5, 8, 9, 20, 7, 2, 12, 16] * 4), (4, [1, 2, 0, 3, 1, 1, 2, 5, 1, 2] * 12)], ids=["few", "one"])
def test_small_keys_in_the_wide_forms(kd, vd, heads, lengths):
    """Keys of at most 32 rows against more than 32 columns: 64 and 128 columns per block, with a last block of few columns."""
    inp = orc.make_inputs(1, sum(lengths), heads, kd, vd, seed=vd, with_state=True, lengths=lengths)
    dev = {n: t.cuda() if torch.is_tensor(t) else t for n, t in inp.items()}
    want_o, want_s = orc.recurrent_kda_ref(*(inp[n].double() for n in ("q", "k", "v", "gate_log2", "beta", "h0")),
                                           inp["cu_seqlens"])
    for call, gate in ((kda_b200.recurrent_kda, "gate_log2"), (kda_b200.chunk_kda, "cum_gate")):
        o, s = call(dev["q"], dev["k"], dev["v"], dev[gate], dev["beta"], dev["h0"], cu_seqlens=dev["cu_seqlens"],
                    output_final_state=True, **({"exact_fp32": True} if gate == "cum_gate" else {}))
        _close(o, want_o, "output")
        _close(s, want_s, "state")


@pytest.mark.parametrize("kd,vd", [(128, 128), (96, 64), (72, 100), (65, 132)])
@pytest.mark.parametrize("lengths", [[4, 1, 0, 3, 5, 8, 9, 20, 7, 2, 12, 16] * 2, [1, 2, 0, 3, 1, 1, 2, 5, 1, 2] * 4], ids=["few", "one"])
def test_many_chains_of_few_tokens(kd, vd, lengths):
    """64 or 32 columns per CTA and tiles of four or two tokens: lengths around these that average under 8 and under 2."""
    inp = orc.make_inputs(1, sum(lengths), 4, kd, vd, seed=kd, with_state=True, lengths=lengths)
    dev = {n: t.cuda() if torch.is_tensor(t) else t for n, t in inp.items()}
    want_o, want_s = orc.recurrent_kda_ref(*(inp[n].double() for n in ("q", "k", "v", "gate_log2", "beta", "h0")),
                                           inp["cu_seqlens"])
    for call, gate in ((kda_b200.recurrent_kda, "gate_log2"), (kda_b200.chunk_kda, "cum_gate")):
        o, s = call(dev["q"], dev["k"], dev["v"], dev[gate], dev["beta"], dev["h0"], cu_seqlens=dev["cu_seqlens"],
                    output_final_state=True, **({"exact_fp32": True} if gate == "cum_gate" else {}))
        _close(o, want_o, "output")
        _close(s, want_s, "state")
