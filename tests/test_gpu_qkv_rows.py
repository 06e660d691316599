"""The chunked pair on rows of q | k | v, as KDAAttention calls it, against the same pair on three tensors: the same
kernels with another pitch, so the same bits; partial chunks (plain loads and stores beside the tensor maps), packed
batches with an unused tail, states and their gradients."""

import pytest
import torch

from kda_b200.chunk_schedule import prepare_ragged_chunk_metadata
from kda_b200.fused import chunk_forward, chunk_forward_qkv

pytestmark = pytest.mark.gpu


def _inputs(batch, tokens, heads, lengths, state, seed=5):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    r = lambda *s: torch.randn(*s, generator=gen, device="cuda")
    qkv = r(batch, tokens, 3, heads, 128).bfloat16()
    gate = -0.3 * torch.rand(batch, tokens, heads, 128, generator=gen, device="cuda")
    marks = [0]
    for n in lengths or [tokens]:
        marks.append(marks[-1] + n)
    for a, b in zip(marks[:-1], marks[1:]):
        for c in range(a, b, 64):
            gate[:, c:min(c + 64, b)] = gate[:, c:min(c + 64, b)].cumsum(1)
    beta = r(batch, tokens, heads).sigmoid()
    nseq = len(lengths) if lengths else batch
    h0 = 0.1 * r(nseq, heads, 128, 128) if state else None
    meta = None
    if lengths:
        meta = prepare_ragged_chunk_metadata(torch.tensor(marks, dtype=torch.int32, device="cuda"), tokens, 64)
    return qkv, gate, beta, h0, meta, r(batch, tokens, heads, 128).bfloat16(), r(nseq, heads, 128, 128)


@pytest.mark.parametrize("batch,tokens,heads,lengths", [
    (1, 1, 1, None), (2, 64, 3, None), (3, 130, 2, None), (1, 8192, 2, None),                 # the last one in segments
    (1, 301, 3, [1, 0, 63, 64, 65, 100]),                                                     # eight tokens unused
])
@pytest.mark.parametrize("state", [False, True])
def test_same_bits_as_three_tensors(batch, tokens, heads, lengths, state):
    qkv, gate, beta, h0, meta, d_out, d_state = _inputs(batch, tokens, heads, lengths, state)
    results = []
    for fused in (False, True):
        leaves = [t.clone().requires_grad_() for t in (qkv, gate, beta, h0) if t is not None]
        x, g, b = leaves[:3]
        h = leaves[3] if state else None
        if fused:
            o, s = chunk_forward_qkv(x, g, b, h, metadata=meta, output_final_state=state)
        else:
            o, s = chunk_forward(*x.unbind(2), g, b, h, metadata=meta, output_final_state=state, normalize_qk=True)
        outs, cots = ([o, s], [d_out, d_state]) if state else ([o], [d_out])
        results.append([*outs, *torch.autograd.grad(outs, leaves, cots)])
    for a, b in zip(*results):
        assert torch.equal(a, b)
    with torch.no_grad():
        o, _ = chunk_forward_qkv(qkv, gate, beta, h0, metadata=meta)
    assert torch.equal(o, results[0][0])


def test_compiler_contract():
    qkv, gate, beta, h0, meta, d_out, d_state = _inputs(1, 150, 2, [70, 80], True)
    ops = torch.ops.kda_b200_layer
    utils = ("test_schema", "test_faketensor")
    for cu, co, h in ((None, None, None), (meta.cu_seqlens, meta.chunk_offsets, h0)):
        args = (qkv, gate, beta, h, cu, co, True, True, 1e-6)
        torch.library.opcheck(ops.chunk_fwd_qkv.default, args, test_utils=utils)
        out, state, aqk, akk, saved, rq, rk = ops.chunk_fwd_qkv(*args)
        d_s = d_state[:state.shape[0]]
        torch.library.opcheck(ops.chunk_bwd_qkv.default, (qkv, gate, beta, aqk, akk, saved, rq, rk, cu, co, d_out, d_s, h,
                                                          h is not None), test_utils=utils)


@pytest.mark.parametrize("bad", ["cpu", "fp32", "shape"])
def test_rejections(bad):
    qkv, gate, beta, *_ = _inputs(1, 64, 1, None, False)
    qkv = {"cpu": lambda: qkv.cpu(), "fp32": lambda: qkv.float(), "shape": lambda: qkv[:, :, :2].contiguous()}[bad]()
    with pytest.raises((ValueError, TypeError, NotImplementedError)):
        chunk_forward_qkv(qkv, gate.cpu() if bad == "cpu" else gate, beta.cpu() if bad == "cpu" else beta)
