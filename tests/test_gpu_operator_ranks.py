"""Operators called directly with q of another rank than four refuse it, as ``batch, tokens, heads, dim = q.shape`` did."""

import pytest
import torch

import kda_b200  # noqa: F401

pytestmark = pytest.mark.gpu
ops = torch.ops.kda_b200


def _inputs(shape):
    q = torch.zeros(shape, device="cuda", dtype=torch.bfloat16)
    gate, beta = torch.zeros(1, 64, 2, 128, device="cuda"), torch.zeros(1, 64, 2, device="cuda")
    return q, gate, beta


@pytest.mark.parametrize("shape", [(1, 64, 2, 128, 1), (64, 2, 128), (1, 64, 2, 1, 128)])
def test_q_of_another_rank(shape):
    q, gate, beta = _inputs(shape)
    tape = torch.zeros(1, 64, 2, 64, device="cuda", dtype=torch.bfloat16)
    saved = torch.zeros(2 ** 24, device="cuda", dtype=torch.uint8)
    rstd = torch.zeros(1, 64, 2, device="cuda")
    calls = (
        lambda: ops.kda_chunk_fwd(q, q, q, gate, beta, None, True),
        lambda: ops.kda_chunk_fwd_saved(q, q, q, gate, beta, None, None, None, False),
        lambda: ops.kda_chunk_bwd_saved(q, q, q, gate, beta, tape, tape, saved, None, None, None, None, None, False),
        lambda: ops.kda_chunk_bwd_qknorm(q, q, q, gate, beta, tape, tape, saved, rstd, rstd, None, None, None, None, None, False),
        lambda: ops.kda_recurrent_fwd(q, q, q, gate, beta, None, None, True),
        lambda: ops.kda_recurrent_fwd_no_state(q, q, q, gate, beta, None, None, True),
    )
    for call in calls:
        with pytest.raises(ValueError):
            call()
