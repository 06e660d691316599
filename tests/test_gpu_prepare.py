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


@pytest.mark.parametrize("sequences", [111, 112, 113, 366, 367, 368])
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


def _tape(k, beta=1.0):
    """(I + L)^-1 of every chunk as the forward pass stores it, for gates of zero: [chunks, H, 64, 64]."""
    tokens, heads = k.shape[1:3]
    gen = torch.Generator().manual_seed(45)
    q, v = (torch.randn(k.shape, generator=gen).bfloat16().cuda() for _ in range(2))
    akk = torch.ops.kda_b200.kda_chunk_fwd(q, k.bfloat16().cuda(), v, torch.zeros(k.shape, device="cuda"),
                                           torch.full(k.shape[:3], beta, device="cuda"), None, True)[2]
    return akk[0].reshape(tokens // 64, 64, heads, 64).transpose(1, 2).double().cpu()


def _inverse_by_blocks(L):
    """(I + L)^-1 by 16 x 16 blocks in the dtype of L: diagonal blocks by substitution, every other block as one
    product, summed in two halves of interleaved groups of four."""
    eye = torch.eye(16, dtype=L.dtype)
    blk = lambda M, r, c: M[..., 16 * r:16 * r + 16, 16 * c:16 * c + 16]
    A = torch.zeros_like(L)
    for b in range(4):
        blk(A, b, b)[:] = torch.linalg.solve_triangular(eye + blk(L, b, b), eye.expand_as(blk(L, b, b)), upper=False)
    for d in range(1, 4):
        half = torch.arange(16 * d) % 8 < 4
        for c in range(4 - d):
            r = c + d
            left = torch.cat([blk(A, r, r) @ blk(L, r, m) for m in range(c, r)], -1)
            right = torch.cat([blk(A, m, c) for m in range(c, r)], -2)
            blk(A, r, c)[:] = -(left[..., half] @ right[..., half, :] + left[..., ~half] @ right[..., ~half, :])
    return A


def test_inverse_keeps_fp32_operands():
    """Equal rows k in a chunk make L = c ones below the diagonal, exact in fp32 (c: a sum of 16-bit squares), and an
    inverse whose entries -c (1 - c)^(d - 1) die out with the distance d: what is stored there is the rounding
    error of the solve, not hidden by the bf16 of the tape.  It is that of fp32 operands, 5.6e-9 (root mean square), up
    to the order of sums of 8 terms (factor 1.2); operands of two tf32 halves give 8.8e-9."""
    gen = torch.Generator().manual_seed(46)
    heads, chunks = 8, 8
    base = torch.randint(1, 32, (chunks, heads, 128), generator=gen) / 256.0
    base = torch.where((base * base).cumsum(-1) < 0.99, base, 0.0)
    k = base[:, None].expand(chunks, 64, heads, 128).reshape(1, chunks * 64, heads, 128)
    c = (base.double() ** 2).sum(-1)[..., None, None]
    L = c * torch.ones(64, 64, dtype=torch.float64).tril(-1)
    assert torch.equal(L.float().double(), L) and torch.equal(k.bfloat16().float(), k)
    want = torch.linalg.inv(torch.eye(64, dtype=torch.float64) + L)
    below = torch.block_diag(*[torch.ones(16, 16)] * 4) == 0
    where = below & (want.abs() < 1e-9) & (torch.ones(64, 64).tril() > 0)
    rms = lambda A: float(((A.double() - want)[where] ** 2).mean().sqrt())
    assert int(where.sum()) > 20000
    assert rms(_tape(k)) <= 1.2 * rms(_inverse_by_blocks(L.float()).bfloat16())


def test_nan_reaches_every_entry_that_depends_on_it():
    gen = torch.Generator().manual_seed(47)
    k = torch.nn.functional.normalize(torch.randn(1, 128, 2, 128, generator=gen), dim=-1)
    k[0, 5, 1, 77] = float("nan")                   # chunk 0, head 1, row 5
    A = _tape(k, 0.5)
    # L has NaN in row 5 and column 5: so has the inverse, in every row below
    assert torch.isnan(A[0, 1, 6:, 5]).all() and torch.isnan(A[0, 1, 5, :5]).all()
    assert torch.isnan(A[0, 1, 6:, :5]).all()
    assert torch.isfinite(A[0, 0]).all() and torch.isfinite(A[1]).all()


def test_gated_query_is_rounded_once():
    """scale q 2^G from one exponential and two fp32 products, bit for bit (torch evaluates the same exp2 in fp32 on
    the device); 2^G as a product of two exponentials differs in one value out of 10^5."""
    tokens, heads = 4096, 8
    gen = torch.Generator(device="cuda").manual_seed(48)
    q, k, v = (torch.randn(1, tokens, heads, 128, generator=gen, device="cuda").bfloat16() for _ in range(3))
    gate = -0.5 * torch.rand(1, tokens, heads, 128, generator=gen, device="cuda")
    gate = gate.unflatten(1, (-1, 64)).cumsum(2).flatten(1, 2)
    beta = torch.full((1, tokens, heads), 0.5, device="cuda")
    saved = torch.ops.kda_b200.kda_chunk_fwd_saved(q, k, v, gate, beta, None, None, None, False)[4]
    n = tokens * heads * 128
    qg = saved[:8 * n].view(torch.bfloat16)[3 * n:].view(q.shape)
    scale = float(torch.tensor(128.0, dtype=torch.float64).rsqrt().float())
    assert torch.equal(qg, (q.float() * torch.exp2(gate) * scale).bfloat16())
