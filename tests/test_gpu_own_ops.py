"""Compiler contract of the operators of the ``kda_b200_fused`` namespace (schema, aliasing and mutation, fake tensors
against the real ones), as test_gpu_opcheck.py has it for ``kda_b200``, and both public calls traced as one graph."""

import pytest
import torch

import kda_b200

pytestmark = pytest.mark.gpu
CHECKS = ("test_schema", "test_faketensor")
ops = torch.ops.kda_b200_fused


def _normal(seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    return gen, lambda *s: torch.randn(*s, generator=gen, device="cuda")


def _scan_args(transposed):
    _, r = _normal(81)
    q, k = (torch.nn.functional.normalize(r(2, 70, 3, 40), dim=-1) for _ in range(2))
    v = r(2, 3, 70, 24).transpose(1, 2) if transposed else r(2, 70, 3, 24)
    return q, k, v, -torch.rand_like(q), r(2, 70, 3).sigmoid(), r(2, 3, 40, 24)


@pytest.mark.parametrize("transposed", [False, True])
def test_scan_operator(transposed):
    args = _scan_args(transposed)
    torch.library.opcheck(ops.chunk_scan.default, (*args, None, True), test_utils=CHECKS)
    cu = torch.tensor([0, 30, 30, 65], dtype=torch.int32, device="cuda")
    one = tuple(t[:1] for t in args[:5])
    torch.library.opcheck(ops.chunk_scan.default, (*one, None, cu, False), test_utils=CHECKS)


def test_scan_traced_as_one_graph():
    args = _scan_args(True)
    with torch.no_grad():
        f = lambda *a: kda_b200.chunk_kda(*a, output_final_state=True)
        for a, b in zip(f(*args), torch.compile(f, fullgraph=True, backend="aot_eager")(*args)):
            assert torch.equal(a, b) and a.stride() == b.stride()


def _decode_args(dtype=torch.bfloat16, width=4):
    gen, r = _normal(82)
    heads, seqs, slots = 2, 3, 5
    idx = torch.tensor([4, 0, 2], dtype=torch.int32, device="cuda")
    return dict(x=r(seqs, 384 * heads).to(dtype), conv_weight=(0.5 * r(384 * heads, width)).to(dtype),
                conv_state=r(slots, width - 1, 384 * heads).to(dtype), raw_gate=r(seqs, heads, 128).to(dtype),
                A_log=0.3 * r(heads), dt_bias=0.3 * r(heads, 128), beta=r(seqs, heads).sigmoid(),
                state_pool=0.02 * r(slots, heads, 128, 128), state_indices=idx)


@pytest.mark.parametrize("dtype,width", [(torch.bfloat16, 4), (torch.float32, 3)])
def test_decode_step_operator(dtype, width):
    a = _decode_args(dtype, width)
    torch.library.opcheck(ops.decode_step.default,
                          (a["x"], a["conv_weight"], a["conv_state"], a["state_pool"], a["state_indices"], a["raw_gate"],
                           a["A_log"], a["dt_bias"], a["beta"], "silu", -5.0, 1e-6), test_utils=CHECKS)


def test_decode_step_traced_as_one_graph():
    eager, traced = _decode_args(), _decode_args()
    with torch.no_grad():
        f = lambda kw: kda_b200.decode_step(**kw)
        compiled = torch.compile(f, fullgraph=True, backend="aot_eager")
        for _ in range(3):
            assert torch.equal(f(eager), compiled(traced))
    for name in ("conv_state", "state_pool"):
        assert torch.equal(eager[name], traced[name]), name


def test_every_operator_of_the_namespace_is_covered():
    registered = {name.split("::")[1].split(".")[0]
                  for name in torch._C._dispatch_get_all_op_names() if name.startswith("kda_b200_fused::")}
    assert registered == {"chunk_scan", "decode_step"}, registered
