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


def _decode_args(slots=3, heads=2, seqs=2):
    def e(*shape, dtype=torch.bfloat16):
        return torch.empty(*shape, dtype=dtype, device="cuda")
    f32 = torch.float32
    return dict(x=e(seqs, 384 * heads), conv_weight=e(384 * heads, 4), conv_state=e(slots, 3, 384 * heads),
                raw_gate=e(seqs, heads, 128), A_log=e(heads, dtype=f32), dt_bias=e(heads, 128, dtype=f32),
                beta=e(seqs, heads, dtype=f32), state_pool=e(slots, heads, 128, 128, dtype=f32),
                state_indices=e(seqs, dtype=torch.int32))


@pytest.mark.parametrize("name", ["x", "conv_weight", "conv_state", "raw_gate", "A_log", "dt_bias", "beta", "state_pool"])
def test_decode_step_refuses_tensors_that_ask_for_gradients(name):
    with FakeTensorMode():
        args = _decode_args()
        args[name].requires_grad_()
        with pytest.raises(RuntimeError, match="inference-only"):
            kda_b200.decode_step(**args)
        with torch.no_grad():
            out = kda_b200.decode_step(**args)
        assert tuple(out.shape) == (2, 2, 128) and out.dtype == torch.bfloat16 and not out.requires_grad


def test_decode_step_refuses_pools_whose_strides_recurrent_kda_refuses():
    with FakeTensorMode(), torch.no_grad():
        args = _decode_args(slots=1)              # an axis of length one may have any stride and count as contiguous
        args["state_pool"] = args["state_pool"].as_strided((1, 2, 128, 128), (16384, 16384, 128, 1))
        with pytest.raises(ValueError, match="overlap"):
            kda_b200.decode_step(**args)
        args = _decode_args(heads=1)
        args["state_pool"] = args["state_pool"].as_strided((3, 1, 128, 128), (16384, 7, 128, 1))
        with pytest.raises(TypeError, match="within each"):
            kda_b200.decode_step(**args)
