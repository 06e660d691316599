"""The bits of a sequence in a scan of 16-bit rows do not depend on the other sequences of the call, from three tokens on: alone (one
column per lane) and in batches that take the wide forms, dense and packed, aligned state rows and others."""

import pytest
import torch

import kda_b200

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kd,vd", [(32, 32), (20, 16), (64, 64), (64, 128), (96, 36), (128, 128), (128, 130)])
@pytest.mark.parametrize("tokens", [3, 7, 10, 33, 70])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_alone_and_in_a_batch(kd, vd, tokens, dtype):
    heads, batch = 4, 160
    gen = torch.Generator(device="cuda").manual_seed(kd + tokens)
    r = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    q, k = (torch.nn.functional.normalize(r(batch, tokens, heads, kd), dim=-1).to(dtype) for _ in range(2))
    v, gate, beta = r(batch, tokens, heads, vd).to(dtype), -r(batch, tokens, heads, kd).abs(), r(batch, tokens, heads).sigmoid()
    h0 = r(batch, heads, kd, vd)
    args = (q, k, v, gate, beta)
    out, state = kda_b200.recurrent_kda(*args, h0, output_final_state=True)
    for n in (1, 9):          # 9: between the lines for most sizes
        o, s = kda_b200.recurrent_kda(*(x[:n].contiguous() for x in args), h0[:n].contiguous(), output_final_state=True)
        assert torch.equal(o, out[:n]) and torch.equal(s, state[:n]), n
    cu = torch.arange(0, batch * tokens + 1, tokens, dtype=torch.int32, device="cuda")
    o, s = kda_b200.recurrent_kda(*(x.reshape(1, batch * tokens, *x.shape[2:]) for x in args), h0, cu_seqlens=cu,
                                  output_final_state=True)
    assert torch.equal(o.view_as(out), out) and torch.equal(s, state)
