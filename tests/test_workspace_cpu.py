"""Workspace sizes of the dense chunked forward (shape-only functions of the library, no GPU needed): a dense batch
takes what the same rows take as a packed batch, plus the offsets, plus three fp32 states per (segment, head) only
where rows really are walked in segments and nothing is kept for a backward pass."""

import pytest

from kda_b200 import _cabi, build

SHAPES = [(1, 1, 1), (2, 130, 2), (1024, 64, 32), (64, 512, 32), (16, 64, 32), (8, 4096, 32), (2, 4096, 32),
          (1, 8191, 4), (1, 8192, 1), (1, 8192, 32), (2, 16384, 8), (1, 131072, 32), (1, 131072, 74), (1, 131072, 75)]


def _sizes(batch, tokens, heads):
    lib = _cabi.lib()
    chunks = batch * ((tokens + 63) // 64)
    return ([lib.kda_chunk_fwd_dense_workspace_bytes(batch, tokens, heads, keep) for keep in (0, 1)],
            lib.kda_chunk_fwd_workspace_bytes(batch * tokens, heads),
            lib.kda_chunk_bwd_workspace_bytes(batch * tokens, heads, chunks))


@pytest.mark.parametrize("batch,tokens,heads", SHAPES)
def test_dense_workspace_is_that_of_packed_rows(batch, tokens, heads):
    build.build()
    (plain, kept), packed, packed_kept = _sizes(batch, tokens, heads)
    assert kept == packed_kept                    # lives until the backward pass: not a byte more
    segments = max(1, min(8, 148 // (batch * heads), ((tokens + 63) // 64) // 64))
    extra = 2 * 4 * (batch * segments + 1) + 3 * 256
    if segments > 1:
        extra += batch * segments * heads * (3 * 128 * 128 * 4 + 4) + 256
    assert packed <= plain <= packed + extra
    assert plain - packed <= 0.05 * packed + 16384          # 192 KiB a segment beside 1 KiB a token of at least 4096


@pytest.mark.parametrize("segments", [2, 12, 64])
def test_forced_segments_have_room(segments):
    build.build()
    lib = _cabi.lib()
    states = 2 * min(segments, 12) * 3 * 3 * 128 * 128 * 4
    try:
        assert lib.kda_set_row_segments(segments) == 0
        (plain, kept), packed, packed_kept = _sizes(2, 64 * 11 + 17, 3)
    finally:
        lib.kda_set_row_segments(0)
    hidden = 2 * 12 * 3 * 128 * 128 * 2           # the chunk states' gradients, free until the backward pass
    assert plain >= packed + states and kept >= packed_kept + (states if states > hidden else 0)
