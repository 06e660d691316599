"""A wait of the state-streaming kernel that runs out: the kernel returns and reports it, no state is left half advanced, and the
next call works.  One warp of each role gives up, at the first state, inside the ring and past one turn of the operand slots."""

import pytest
import torch

import kda_b200
from kda_b200 import _cabi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("warp", [0, 3, 6, 15, 16, 17, 20, 22])
@pytest.mark.parametrize("step", [0, 2, 9])
def test_a_wait_that_runs_out(warp, step):
    lib = _cabi.lib()
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    n = 12 * sms + 5                                    # the first block takes states 0, sms, 2 sms, ..
    gen = torch.Generator(device="cuda").manual_seed(warp + step)
    q, k, v = (torch.nn.functional.normalize(torch.randn(n, 128, generator=gen, device="cuda"), dim=-1) for _ in range(3))
    gate, beta = -torch.rand(n, 128, generator=gen, device="cuda"), torch.rand(n, generator=gen, device="cuda")
    before = torch.randn(n, 128, 128, generator=gen, device="cuda")

    def whole():
        rows = [x.view(n, 1, 1, 128) for x in (q, k, v, gate)]
        return kda_b200.recurrent_kda(*rows, beta.view(n, 1, 1), before.view(n, 1, 128, 128),
                                      output_final_state=True)[1].view(n, 128, 128)

    want = whole()
    torch.cuda.synchronize()
    assert lib.kda_device_error_word() == 0
    states, out = before.clone(), torch.empty(n, 128, device="cuda")
    assert lib.kda_selftest_bounded_stream(*(x.data_ptr() for x in (q, k, v, gate, beta, states, out)), n, warp, step,
                                           _cabi.stream()) == 0
    torch.cuda.synchronize()
    assert lib.kda_device_error_word() == 64 and lib.kda_device_error_word() == 0
    kept, advanced = (states == before).flatten(1).all(1), (states == want).flatten(1).all(1)
    assert (kept | advanced).all()
    first = torch.zeros(n, dtype=torch.bool, device="cuda")
    first[::sms] = True
    assert advanced[~first].all()                       # the other blocks
    # (an operand warp takes every third state; earlier states may be given up too, except by the copying warp itself)
    last = step if warp <= 16 else step + 2
    assert kept[::sms][last:].all()
    if warp == 16:
        assert advanced[::sms][:step].all()
    assert torch.equal(whole(), want) and lib.kda_device_error_word() == 0


def test_arguments():
    assert _cabi.lib().kda_selftest_bounded_stream(*([None] * 7), 1, 0, 0, None) == -1
