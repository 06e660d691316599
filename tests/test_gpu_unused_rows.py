"""Rows of packed results that no sequence covers are zero, whatever their memory held: every operator that takes packed
offsets, forward and backward, with an unused tail of one row, of many and of none, more sequences than a block has
threads, odd row sizes, and offsets that the kernels skip."""

import ctypes

import pytest
import torch

import kda_b200
from kda_b200 import _cabi
from kda_b200.chunk_schedule import prepare_ragged_chunk_metadata

pytestmark = pytest.mark.gpu


def _poison():
    """Freed blocks of every size class hold NaN, so that an element nobody writes shows."""
    held = [torch.full((n,), float("nan"), device="cuda") for n in (128, 2 ** 10, 2 ** 14, 2 ** 18, 2 ** 20, 2 ** 22, 2 ** 24)
            for _ in range(4)]
    del held


@pytest.mark.parametrize("lengths,unused", [([5], 1), ([64, 0, 63], 70), ([1] * 300, 3), ([100, 28], 0)], ids=str)
@pytest.mark.parametrize("normalize", [False, True])
def test_core(lengths, unused, normalize):
    heads, used = 3, sum(lengths)
    tokens = used + unused
    gen = torch.Generator(device="cuda").manual_seed(1)
    r = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    marks = [0]
    for n in lengths:
        marks.append(marks[-1] + n)
    cu = torch.tensor(marks, dtype=torch.int32, device="cuda")
    # keys of unit length: with beta * |k|^2 <= 1 no factor I - beta k k^T grows the state, so every result stays finite
    q, k, v, d = (torch.nn.functional.normalize(r(1, tokens, heads, 128), dim=-1).bfloat16() for _ in range(4))
    gate, beta = -torch.rand(1, tokens, heads, 128, generator=gen, device="cuda"), r(1, tokens, heads).sigmoid()
    leaves = [x.requires_grad_() for x in (q, k, v, gate, beta)]
    for recompute in (False, True)[:1 if normalize else 2]:
        _poison()
        o, _ = kda_b200.chunk_kda(*leaves, cu_seqlens=cu, normalize_qk=normalize, recompute=recompute)
        _poison()
        grads = torch.autograd.grad([o], leaves, [d])
        for x in (o, *grads):
            assert torch.isfinite(x.float()).all() and not x[:, used:].any()
    _poison()
    with torch.no_grad():
        o2, _ = kda_b200.chunk_kda(*leaves, cu_seqlens=cu, normalize_qk=normalize)
    assert torch.equal(o2, o)


@pytest.mark.parametrize("lengths,unused", [([5], 1), ([64, 0, 63], 70), ([1] * 300, 3)], ids=str)
def test_gate_and_convolution(lengths, unused):
    heads, used = 3, sum(lengths)
    tokens = used + unused
    gen = torch.Generator(device="cuda").manual_seed(2)
    r = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    cu = torch.tensor([sum(lengths[:i]) for i in range(len(lengths) + 1)], dtype=torch.int32, device="cuda")
    raw, a_log, bias = r(1, tokens, heads, 128).bfloat16().requires_grad_(), r(heads), r(heads, 128)
    for chunk in (64, 16):
        _poison()
        out = kda_b200.bounded_gate_cumsum(raw, a_log, bias, cu_seqlens=cu, chunk_size=chunk)
        _poison()
        (grad,) = torch.autograd.grad([out], [raw], [torch.ones_like(out)])
        for x in (out, grad):
            assert torch.isfinite(x.float()).all() and not x[:, used:].any()
    for dtype, width, channels in ((torch.bfloat16, 4, 40), (torch.float32, 3, 40), (torch.bfloat16, 2, 8)):
        x, w = r(1, tokens, channels).to(dtype).requires_grad_(), r(channels, width).to(dtype)
        _poison()
        y = kda_b200.causal_conv1d(x, w, activation="silu", cu_seqlens=cu)
        _poison()
        (grad,) = torch.autograd.grad([y], [x], [torch.ones_like(y)])
        for t in (y, grad):
            assert torch.isfinite(t.float()).all() and not t[:, used:].any()


@pytest.mark.parametrize("offsets,chunks,kept", [
    ([0, 70, 90], [0, 2, 3], range(0, 90)), ([3, 70, 90], [0, 2, 3], range(3, 90)),
    ([0, 70, 101], [0, 2, 3], range(0)), ([0, 80, 70], [0, 2, 2], range(0)), ([-1, 70, 90], [0, 2, 3], range(0)),
    ([0, 70, 90], [0, 2, 4], range(0)), ([0, 70, 90], [1, 3, 4], range(0)), ([0, 70, 90], None, range(0, 90)),
], ids=str)
def test_which_rows_are_cleared(offsets, chunks, kept):
    """100 rows of 16, 12, 4, 2 and 10 bytes; offsets that leave the buffer or contradict one another clear everything."""
    buffers = [torch.ones(100, n, device="cuda", dtype=t)
               for n, t in ((4, torch.float32), (3, torch.float32), (1, torch.float32), (1, torch.bfloat16), (5, torch.bfloat16))]
    cu = torch.tensor(offsets, dtype=torch.int32, device="cuda")
    co = torch.tensor(chunks, dtype=torch.int32, device="cuda") if chunks else None
    ptrs = (ctypes.c_void_p * 5)(*(b.data_ptr() for b in buffers))
    sizes = (ctypes.c_int64 * 5)(16, 12, 4, 2, 10)
    _cabi.call("kda_zero_unused_rows", 1, ctypes.addressof(ptrs), ctypes.addressof(sizes), 5, cu.data_ptr(), _cabi.ptr(co),
               64, 2, 100, _cabi.stream())
    want = torch.zeros(100, dtype=torch.bool)
    want[list(kept)] = True
    for b in buffers:
        assert torch.equal(b.cpu().bool().all(1), want) and torch.equal(b.cpu().bool().any(1), want)


@pytest.mark.parametrize("rows", [-1, 0, 1])
def test_where_clearing_rows_replaces_the_fill(rows):
    """Either side of the size from which only the unused rows are cleared: zero there, one more launch beyond it."""
    from kda_b200 import ops

    tokens = ops._FILL_BYTES // (2 * 128 * 4) + rows
    cu = torch.tensor([0, 100, tokens - 70], dtype=torch.int32, device="cuda")
    raw = torch.randn(1, tokens, 2, 128, device="cuda").bfloat16()
    a_log, bias = torch.zeros(2, device="cuda"), torch.zeros(2, 128, device="cuda")
    kda_b200.bounded_gate_cumsum(raw, a_log, bias, cu_seqlens=cu)
    _poison()
    before = _cabi.launch_count
    out = kda_b200.bounded_gate_cumsum(raw, a_log, bias, cu_seqlens=cu)
    launches = _cabi.launch_count - before
    assert torch.isfinite(out).all() and not out[:, -70:].any() and out[:, :-70].any(-1).all()
    assert launches == (3 if rows > 0 else 2)            # the chunk offsets, the gate, and the clearing
