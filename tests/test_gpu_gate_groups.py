"""The backward of the gate where the number of chunks that a block takes changes (96 / 97, 192 / 193 chunks) and where the
last block has fewer chunks than the others, dense and packed, against the fp64 gradients."""

import pytest
import torch

import kda_b200
from oracle import kda_oracle as orc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("chunks", [1, 2, 95, 96, 97, 191, 192, 193, 195])
@pytest.mark.parametrize("packed", [False, True])
def test_chunks_of_a_block(chunks, packed):
    tokens, heads = 16 * chunks - 5, 2
    offsets = torch.tensor([0, 16 * (chunks // 2), tokens], dtype=torch.int32) if packed and chunks > 1 else None
    gen = torch.Generator().manual_seed(chunks)
    raw, d = (torch.randn(1, tokens, heads, 128, generator=gen) for _ in range(2))
    raw = raw.bfloat16()
    a_log, bias = 0.1 * torch.randn(heads, generator=gen), 0.1 * torch.randn(heads, 128, generator=gen)
    want = orc.bounded_gate_cumsum_bwd_ref(raw.double(), a_log.double(), bias.double(), d.double(), 16, -5.0, offsets)
    leaves = [t.cuda().requires_grad_() for t in (raw, a_log, bias)]
    out = kda_b200.bounded_gate_cumsum(*leaves, chunk_size=16, cu_seqlens=None if offsets is None else offsets.cuda())
    got = torch.autograd.grad([out], leaves, [d.cuda()])
    for name, g, w in zip(("raw", "A_log", "dt_bias"), got, want):
        # fp32 sums of `tokens` terms (times 128 channels for A_log) that cancel like a random walk, and 2-ulp intrinsics
        terms = 16 if name == "raw" else tokens * (128 if name == "A_log" else 1)
        bound = 2.0 ** -20 * max(terms, 16) ** 0.5 + (2.0 ** -8 if name == "raw" else 0.0)     # d_raw is bf16
        err = float((g.double().cpu() - w).abs().max() / w.abs().max())
        assert err < bound, (name, err, bound)
