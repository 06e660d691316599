"""h_out = M h_in + b at the edges of its slabs of K, for matrices that start off 16-byte addresses, against fp64."""

import pytest
import torch

from kda_b200 import _cabi

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
