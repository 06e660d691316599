"""The decode operator, called directly, on pools whose slots overlap while the states of the call do not, and on a pool of one slot
with any stride: the results of a packed pool, in one launch and in two."""

import pytest
import torch

import kda_b200  # noqa: F401

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype,width", [(torch.bfloat16, 4), (torch.float16, 2), (torch.bfloat16, 5), (torch.float32, 4)])
@pytest.mark.parametrize("stride", [2 * 16384, 16384 + 4, 16384 + 2])
def test_overlapping_slots(dtype, width, stride):
    heads, slots, at = 3, 4, 2
    gen = torch.Generator(device="cuda").manual_seed(width)
    r = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    x, w = r(1, 3 * heads * 128).to(dtype), r(3 * heads * 128, width).to(dtype)
    conv, raw = r(slots, width - 1, 3 * heads * 128).to(dtype), r(1, heads, 128).to(dtype)
    a_log, bias, beta = r(heads), r(heads, 128), r(1, heads).sigmoid()
    idx = torch.tensor([at], dtype=torch.int32, device="cuda")
    storage = r((slots - 1) * stride + heads * 16384)
    pool = storage.as_strided((slots, heads, 128, 128), (stride, 16384, 128, 1))
    packed, conv2 = pool.contiguous(), conv.clone()
    want = storage.clone()
    step = torch.ops.kda_b200_fused.decode_step
    out2 = step(x, w, conv2, packed, idx, raw, a_log, bias, beta, "silu", -5.0, 1e-6)
    want[at * stride:at * stride + heads * 16384] = packed[at].reshape(-1)
    out = step(x, w, conv, pool, idx, raw, a_log, bias, beta, "silu", -5.0, 1e-6)
    if dtype == torch.float32 or width > 4 or stride % 4:        # other kernels than those of the packed pool: another order of sums
        assert torch.allclose(out.float(), out2.float(), atol=2.0 ** -7 * float(out2.abs().max()))
        assert float((storage - want).abs().max()) < 1e-5 * float(want.abs().max())
    else:
        assert torch.equal(out, out2) and torch.equal(storage, want)
    assert torch.equal(conv, conv2)
