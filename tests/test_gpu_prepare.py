"""The chunk-parallel forward kernel where its tiles end: row blocks of 16, chunks of 64, the number of
sequences whose offsets it keeps in shared memory, several work items per CTA, and a triangular solve of
nearly equal keys (the largest inverse entries).  Tolerance: that of the chunked path, 2e-2 of the largest
oracle value (bf16 operands in several stages), or what bf16 operands cost the oracle itself."""

import pytest
import torch

import kda_b200
from oracle import kda_oracle as orc
from helpers import assert_normalised, norm_err

pytestmark = pytest.mark.gpu
TOL = 2e-2

EDGES = [1, 15, 16, 17, 31, 33, 47, 48, 49, 63, 64, 65, 79, 80, 81, 127, 128, 129]


def _check(inp, normalize=False, budget=False):
    q, k, v = (inp[n].bfloat16() for n in ("q", "k", "v"))
    cu = inp["cu_seqlens"]
    o, st = kda_b200.chunk_kda(q.cuda(), k.cuda(), v.cuda(), inp["cum_gate"].cuda(), inp["beta"].cuda(),
                               None if inp["h0"] is None else inp["h0"].cuda(),
                               cu_seqlens=None if cu is None else cu.cuda(), output_final_state=True,
                               normalize_qk=normalize)
    qf, kf = q.float(), k.float()
    if normalize:
        qf, kf = (x * torch.rsqrt((x * x).sum(-1, keepdim=True) + 1e-6) for x in (qf, kf))
    ref_o, ref_s = orc.chunk_kda_ref(qf, kf, v.float(), inp["cum_gate"], inp["beta"], inp["h0"], cu)
    tol_o = tol_s = TOL
    if budget:       # twice the error of the oracle with bf16 operands, plus two roundings of the result
        low_o, low_s = orc.chunk_kda_ref(qf, kf, v.float(), inp["cum_gate"], inp["beta"], inp["h0"], cu,
                                         store_dtype=torch.bfloat16)
        tol_o, tol_s = (2 * norm_err(x, y) + 2 * 2.0 ** -8 for x, y in ((low_o, ref_o), (low_s, ref_s)))
    assert_normalised(o, ref_o, tol_o, "o")
    assert_normalised(st, ref_s, tol_s, "state")


@pytest.mark.parametrize("normalize", [False, True])
def test_lengths_around_row_blocks_and_chunks(normalize):
    _check(orc.make_inputs(1, sum(EDGES), 2, 128, 128, seed=41, with_state=True, lengths=EDGES), normalize)


@pytest.mark.parametrize("sequences", [111, 112, 113])
def test_sequence_counts_around_the_offset_cache(sequences):
    lengths = [1 + (7 * i) % 23 for i in range(sequences)]
    lengths[sequences // 2] = 0
    _check(orc.make_inputs(1, sum(lengths), 1, 128, 128, seed=42, with_state=True, lengths=lengths))


def test_more_work_items_than_resident_blocks():
    lengths = [64 * 20 + 5, 64 * 13, 3]
    _check(orc.make_inputs(1, sum(lengths), 10, 128, 128, seed=43, with_state=True, lengths=lengths))


def test_nearly_equal_keys():
    inp = orc.make_inputs(1, 192, 2, 128, 128, seed=44, with_state=True)
    inp["k"] = torch.nn.functional.normalize(inp["k"][:, :1] + 0.02 * inp["k"], dim=-1)
    inp["beta"] = torch.full_like(inp["beta"], 0.98)
    inp["cum_gate"] = inp["cum_gate"] * 1e-3
    # the rows of the inverse nearly cancel, and with them the bf16 operands' roundings weigh more than 2e-2
    # of the result: judged by what bf16 operands do to the oracle
    _check(inp, budget=True)
