"""A state that holds infinities at the end of a sequence comes out as the recurrence leaves it, whatever the length of the last block
of the fp32 scan: an infinite value in the last token, and an infinite entering state whose row the keys do not touch."""

import pytest
import torch

import kda_b200
from oracle import kda_oracle as orc

pytestmark = pytest.mark.gpu


def _same(got, want):
    got, want = got.double().cpu(), want.double()
    assert torch.equal(torch.isnan(got), torch.isnan(want))
    assert torch.equal(torch.isinf(got), torch.isinf(want)) and torch.equal(got[torch.isinf(got)], want[torch.isinf(want)])
    finite = torch.isfinite(want)
    assert (got - want)[finite].abs().max() < 1e-4 * want[finite].abs().max()


@pytest.mark.parametrize("tokens", [1, 2, 3, 4, 5, 6, 7, 8, 9, 35])
@pytest.mark.parametrize("kd,vd", [(32, 16), (64, 40), (128, 128)])
@pytest.mark.parametrize("cumulative", [False, True])
def test_infinite_last_value(tokens, kd, vd, cumulative):
    inp = orc.make_inputs(1, tokens, 2, kd, vd, seed=tokens, with_state=True)
    inp["v"][:, -1, :, 3] = float("inf")
    want_o, want_s = orc.recurrent_kda_ref(*(inp[n].double() for n in ("q", "k", "v", "gate_log2", "beta", "h0")))
    args = [inp[n].cuda() for n in ("q", "k", "v", "cum_gate" if cumulative else "gate_log2", "beta", "h0")]
    if cumulative:
        o, s = kda_b200.chunk_kda(*args, output_final_state=True, exact_fp32=True)
    else:
        o, s = kda_b200.recurrent_kda(*args, output_final_state=True)
    _same(s, want_s)
    assert torch.isinf(s[..., 3]).all()
    # (the last output is a sum of infinities of both signs: NaN in one order, infinite in another)
    assert torch.equal(torch.isfinite(o).cpu(), torch.isfinite(want_o))
