"""h_out = M h_in + b at the edges of its slabs of K, for matrices that start off 16-byte addresses, against fp64; and the chain of
such maps along the segments of a row, with and without entering and leaving states, 16 and 32 columns per block."""

import pytest
import torch

import kda_b200
from kda_b200 import _cabi
from oracle import kda_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kd", [64, 128, 192, 256, 320])
@pytest.mark.parametrize("vd", [64, 128, 192])
@pytest.mark.parametrize("offset", [0, 1])
def test_affine(kd, vd, offset):
    count = 3
    gen = torch.Generator(device="cuda").manual_seed(kd + vd)
    m = torch.randn(count * kd * kd + offset, generator=gen, device="cuda")[offset:]
    h = torch.randn(count * kd * vd + offset, generator=gen, device="cuda")[offset:]
    b = torch.randn(count, kd, vd, generator=gen, device="cuda")
    out = torch.full((count, kd, vd), float("nan"), device="cuda")
    _cabi.call("kda_state_affine", 1, m.data_ptr(), h.data_ptr(), b.data_ptr(), out.data_ptr(), count, kd, vd, _cabi.stream())
    m64, h64 = m.view(count, kd, kd).double(), h.view(count, kd, vd).double()
    want = m64 @ h64 + b.double()
    # kd fused multiply-adds and one addition, each rounded to 2^-24 of a partial sum of absolute values
    bound = (kd + 1) * 2.0 ** -24 * (m64.abs() @ h64.abs() + b.double().abs())
    assert ((out.double() - want).abs() <= bound).all()


@pytest.mark.parametrize("segments", [2, 3, 5])
@pytest.mark.parametrize("initial,final", [(True, True), (True, False), (False, True), (False, False)])
def test_chain_of_segments(segments, initial, final):
    """The boundary states of two rows through all their segments, with gates that hardly forget, against the serial walk."""
    inp = orc.make_inputs(2, 64 * 12 - 7, 3, 128, 128, seed=segments, with_state=True)
    q, k, v = (inp[n].bfloat16().cuda() for n in ("q", "k", "v"))
    gate, beta = 0.02 * inp["cum_gate"].cuda(), inp["beta"].cuda()
    h0 = inp["h0"].cuda() if initial else None

    def run(forced):
        try:
            assert _cabi.lib().kda_set_row_segments(forced) == 0
            return kda_b200.chunk_kda(q, k, v, gate, beta, h0, output_final_state=final)
        finally:
            _cabi.lib().kda_set_row_segments(0)

    serial, split = run(1), run(segments)
    # two bf16 evaluations of the products of up to twelve chunks: a few roundings of 2^-9 of the largest value
    for x, y in zip(split[:2 if final else 1], serial):
        assert float((x.double() - y.double()).abs().max() / y.double().abs().max()) < 1e-2


@pytest.mark.parametrize("rows,heads", [(1, 32), (2, 10)])
@pytest.mark.parametrize("segments", [2, 5])
def test_both_widths_of_the_chain(rows, heads, segments):
    """Many chains take 32 columns per block, two rows per thread, few 16.  Both add in the order of K: the first three heads of the large
    call have the bits of a call of their own, and it agrees with the serial walk."""
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert rows * heads * 8 > sms >= rows * 3 * 8
    inp = orc.make_inputs(rows, 64 * 12 - 7, heads, 128, 128, seed=heads, with_state=True)
    q, k, v = (inp[n].bfloat16().cuda() for n in ("q", "k", "v"))
    args = (q, k, v, 0.02 * inp["cum_gate"].cuda(), inp["beta"].cuda(), inp["h0"].cuda())

    def run(forced, some):
        part = [x[:, :, :some].contiguous() for x in args[:5]] + [args[5][:, :some].contiguous()]
        try:
            assert _cabi.lib().kda_set_row_segments(forced) == 0
            return kda_b200.chunk_kda(*part, output_final_state=True)
        finally:
            _cabi.lib().kda_set_row_segments(0)

    (out, state), (few, few_state), serial = run(segments, heads), run(segments, 3), run(1, heads)
    assert torch.equal(out[:, :, :3], few) and torch.equal(state[:, :3], few_state)
    for x, y in zip((out, state), serial):
        assert float((x.double() - y.double()).abs().max() / y.double().abs().max()) < 1e-2
