"""Host side of the two operators of the ``kda_b200_fused`` namespace and of the call that leads to them, on fake CUDA
tensors (no GPU needed): what the registered meta implementations promise, and which calls are refused."""

import pytest
import torch
from torch._subclasses.fake_tensor import FakeTensorMode

import kda_b200


@pytest.mark.parametrize("layout", ["contiguous", "heads_first", "channels_strided"])
def test_scan_result_is_contiguous_whatever_the_layout_of_v(layout):
    batch, tokens, heads, kd, vd = 2, 70, 3, 40, 24
    with FakeTensorMode(), torch.no_grad():
        q, k, g = (torch.empty(batch, tokens, heads, kd, device="cuda") for _ in range(3))
        beta = torch.empty(batch, tokens, heads, device="cuda")
        v = {"contiguous": lambda: torch.empty(batch, tokens, heads, vd, device="cuda"),
             "heads_first": lambda: torch.empty(batch, heads, tokens, vd, device="cuda").transpose(1, 2),
             "channels_strided": lambda: torch.empty(batch, tokens, heads, 2 * vd, device="cuda")[..., ::2]}[layout]()
        out, state = kda_b200.chunk_kda(q, k, v, g, beta, output_final_state=True)
        assert out.shape == v.shape and out.is_contiguous()
        assert tuple(state.shape) == (batch, heads, kd, vd) and state.is_contiguous()
