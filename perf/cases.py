"""Workloads of the KDA path through the package's public entry points, from one decoded token of
one conversation to a packed training batch of 64 sequences.

Families (``kind``):

* ``decode``  one generated token per sequence through ``decode_step`` (short convolution, SiLU,
  l2norm, gate, paged state update), both pools advanced in place;
* ``extend``  a few tokens per sequence through the paged ``recurrent_kda`` (checking drafted tokens,
  the short tails of prompts);
* ``scan``    the fp32-accurate evaluation of ``chunk_kda`` at a head size the chunked kernels do not
  take, for accuracy checks;
* ``prefill`` ``chunk_kda`` without autograd, dense or packed;
* ``train``   ``chunk_kda`` forward + backward, dense or packed;
* ``layer``   ``KDAAttention`` forward + backward, all projections included.

Values are those of the repository's benchmark: q, k ~ N(0, 1) with L2-normalised rows, v ~ N(0, 1),
log-gates ``decay * logsigmoid(N(0, 1))``, beta = sigmoid(N(0, 1)), states ~ N(0, 0.02).  ``decay`` 1.0
forgets a state within a few chunks, 0.02 keeps it over thousands of tokens, as the slow heads of a
trained model do.
"""

import math
import os
import random
import sys

import torch

_PACKAGE = os.path.join(os.getcwd(), "attention-gym_b200")
if _PACKAGE not in sys.path:
    sys.path.insert(1, _PACKAGE)

import kda_b200  # noqa: E402

D = 128                      # head size of the chunked kernels
CHUNK = 64
LOG2E = math.log2(math.e)


def listed():
    return [
        # one conversation, one token: launch and host latency
        {"name": "decode_1", "kind": "decode", "sequences": 1, "heads": 32},
        # a partly filled serving batch
        {"name": "decode_37", "kind": "decode", "sequences": 37, "heads": 32},
        # a full serving batch: the fp32 state pool streams through HBM
        {"name": "decode_256", "kind": "decode", "sequences": 256, "heads": 32},
        # a serving batch in which every sequence brings 1 to 8 tokens
        {"name": "extend_48", "kind": "extend", "sequences": 48, "tokens": 215, "heads": 32},
        # the fp32 check run of a small head size
        {"name": "scan_fp32", "kind": "scan", "batch": 1, "tokens": 512, "heads": 4, "dim": 64},
        # one prompt of ordinary length, its state handed to decoding
        {"name": "prefill_1000", "kind": "prefill", "sequences": 0, "batch": 1, "tokens": 1000,
         "heads": 32, "decay": 0.02, "state": False, "normalize": True},
        # continued prompts of many users packed into one call, states in and out
        {"name": "prefill_packed", "kind": "prefill", "sequences": 16, "batch": 1, "tokens": 40003,
         "heads": 32, "decay": 0.02, "state": True, "normalize": True},
        # one long document
        {"name": "prefill_131072", "kind": "prefill", "sequences": 0, "batch": 1, "tokens": 131072,
         "heads": 32, "decay": 1.0, "state": False, "normalize": False},
        # a small model's step, tail chunk included
        {"name": "train_small", "kind": "train", "sequences": 0, "batch": 2, "tokens": 777, "heads": 8,
         "decay": 1.0, "state": False, "normalize": False, "recompute": False},
        # the headline training step
        {"name": "train_4096", "kind": "train", "sequences": 0, "batch": 8, "tokens": 4096, "heads": 32,
         "decay": 1.0, "state": False, "normalize": False, "recompute": False},
        # a packed training batch with entering states and their gradients
        {"name": "train_packed", "kind": "train", "sequences": 64, "batch": 1, "tokens": 279046,
         "heads": 32, "decay": 1.0, "state": True, "normalize": False, "recompute": False},
        # one whole layer's training step
        {"name": "layer_4096", "kind": "layer", "sequences": 0, "batch": 2, "tokens": 4096, "heads": 32,
         "hidden": 4096},
    ]


def _log_uniform(rng, low, high):
    return min(high, max(low, round(math.exp(rng.uniform(math.log(low), math.log(high))))))


def draw(rng: random.Random):
    kind = rng.choice(("decode", "extend", "scan", "prefill", "prefill", "train", "train", "layer"))
    heads = rng.choice((4, 6, 8, 12, 16, 24, 32))
    if kind == "decode":
        return {"kind": kind, "sequences": _log_uniform(rng, 1, 256), "heads": heads}
    if kind == "extend":
        n = _log_uniform(rng, 1, 128)
        return {"kind": kind, "sequences": n, "tokens": n * rng.randint(2, 7) + rng.randint(0, n), "heads": heads}
    if kind == "scan":
        return {"kind": kind, "batch": rng.randint(1, 4), "tokens": _log_uniform(rng, 64, 1024),
                "heads": rng.randint(1, 8), "dim": rng.choice((32, 64, 96))}
    if kind == "layer":
        heads = rng.choice((4, 8, 16, 32))
        packed = rng.random() < 0.5
        tokens = _log_uniform(rng, 128, 8192)
        batch = 1 if packed else rng.randint(1, max(1, min(4, 8192 // tokens)))
        return {"kind": kind, "sequences": rng.randint(1, max(1, tokens // 64)) if packed else 0,
                "batch": batch, "tokens": tokens, "heads": heads, "hidden": 128 * heads}
    # prefill and train: up to 4 M and 8 M (token, head) pairs, no more work than the largest listed
    # cases; one sequence has at most as many tokens as the longest listed one
    units = _log_uniform(rng, 2000, 4_000_000 if kind == "prefill" else 8_000_000)
    packed = rng.random() < 0.5
    total = max(1, units // heads)
    if packed:
        sequences = _log_uniform(rng, 1, max(1, min(96, total // 64)))
        batch, tokens = 1, min(total, 65536 * sequences)
    else:
        sequences, batch = 0, _log_uniform(rng, 1, max(1, min(16, total // 64)))
        tokens = min(131072, total // batch)
    case = {"kind": kind, "sequences": sequences, "batch": batch, "tokens": tokens, "heads": heads,
            "decay": rng.choice((1.0, 0.02)), "state": rng.random() < 0.5, "normalize": rng.random() < 0.4}
    if kind == "train":
        case["recompute"] = not case["normalize"] and rng.random() < 0.25
    return case


class _Values:
    """Seeded tensors on the GPU."""

    def __init__(self, seed):
        self.gen = torch.Generator(device="cuda").manual_seed(int(seed))
        self.rng = random.Random(int(seed))

    def normal(self, *shape, scale=1.0, dtype=torch.float32):
        x = torch.randn(*shape, generator=self.gen, device="cuda")
        return (x.mul_(scale) if scale != 1.0 else x).to(dtype)

    def rows(self, *shape, unit=True, dtype=torch.bfloat16):
        x = torch.randn(*shape, generator=self.gen, device="cuda")
        return (torch.nn.functional.normalize(x, dim=-1) if unit else x).to(dtype)

    def log_gate(self, *shape, decay=1.0):
        x = torch.randn(*shape, generator=self.gen, device="cuda")
        return torch.nn.functional.logsigmoid(x).mul_(LOG2E * decay)

    def beta(self, *shape):
        return torch.randn(*shape, generator=self.gen, device="cuda").sigmoid_()

    def lengths(self, sequences, tokens):
        """`sequences` positive lengths that add up to `tokens`, the longest up to 64 times the shortest."""
        weights = [self.rng.uniform(1.0, 64.0) for _ in range(sequences)]
        spare, total = tokens - sequences, sum(weights)
        marks, acc = [0], 0.0
        for i, w in enumerate(weights):
            acc += w
            marks.append(i + 1 + int(round(spare * acc / total)))
        marks[-1] = tokens
        return marks


def _cumulative(gate, offsets=None):
    """Prefix sums inside 64-token chunks (in place), restarting at every row and sequence."""
    tokens = gate.shape[1]
    marks = [0, tokens] if offsets is None else offsets
    for a, b in zip(marks[:-1], marks[1:]):
        whole = (b - a) // CHUNK * CHUNK
        if whole:
            part = gate[:, a:a + whole].unflatten(1, (-1, CHUNK))
            part.copy_(part.cumsum(2))
        if whole < b - a:
            part = gate[:, a + whole:b]
            part.copy_(part.cumsum(1))
    return gate


def prepare(case, seed):
    val, kind, heads = _Values(seed), case["kind"], case["heads"]
    bf16 = torch.bfloat16
    state = {"case": case}
    if kind == "decode":
        n, width = case["sequences"], 3 * heads * D
        state.update(
            x=val.normal(n, width, dtype=bf16), weight=val.normal(width, 4, scale=0.5, dtype=bf16),
            conv=val.normal(n + 1, 3, width, dtype=bf16), raw=val.normal(n, heads, D, dtype=bf16),
            a_log=val.normal(heads, scale=0.1), bias=val.normal(heads, D, scale=0.1),
            beta=val.beta(n, heads), pool=val.normal(n + 1, heads, D, D, scale=0.02),
            slots=torch.randperm(n, generator=val.gen, device="cuda").int() + 1)
        return state
    if kind == "extend":
        n, t = case["sequences"], case["tokens"]
        shape = (1, t, heads, D)
        # 1 to 8 tokens for each sequence
        counts, left = [1] * n, t - n
        while left:
            i = val.rng.randrange(n)
            if counts[i] < 8:
                counts[i] += 1
                left -= 1
        marks = [0]
        for c in counts:
            marks.append(marks[-1] + c)
        state.update(
            q=val.rows(*shape), k=val.rows(*shape), v=val.normal(*shape, dtype=bf16),
            gate=val.log_gate(*shape), beta=val.beta(1, t, heads),
            pool=val.normal(n + 1, heads, D, D, scale=0.02),
            cu=torch.tensor(marks, dtype=torch.int32, device="cuda"),
            slots=torch.randperm(n, generator=val.gen, device="cuda").int() + 1)
        return state
    if kind == "scan":
        shape = (case["batch"], case["tokens"], heads, case["dim"])
        state.update(
            q=val.rows(*shape, dtype=torch.float32), k=val.rows(*shape, dtype=torch.float32),
            v=val.normal(*shape), gate=_cumulative(val.log_gate(*shape)), beta=val.beta(*shape[:3]))
        return state
    batch, tokens, sequences = case["batch"], case["tokens"], case["sequences"]
    marks = val.lengths(sequences, tokens) if sequences else None
    state["cu"] = torch.tensor(marks, dtype=torch.int32, device="cuda") if marks else None
    if kind == "layer":
        torch.manual_seed(int(seed))
        layer = kda_b200.KDAAttention(case["hidden"], heads, D, device="cuda")
        with torch.no_grad():
            # gates of a trained layer: decays from 0.1 % to a few per cent a token.  (With a zero bias a
            # state is gone within a chunk, and the gradients of the gate parameters are sums that
            # cancel down to the rounding of their bf16 terms.)
            layer.A_log.copy_(val.normal(heads, scale=0.3))
            layer.dt_bias.copy_(val.normal(heads, D).sub_(5.0))
        state.update(layer=layer, params=list(layer.parameters()),
                     x=val.normal(batch, tokens, case["hidden"], dtype=bf16).requires_grad_(),
                     d_out=val.normal(batch, tokens, case["hidden"], dtype=bf16))
        return state
    shape = (batch, tokens, heads, D)
    unit = not case["normalize"]
    state.update(
        q=val.rows(*shape, unit=unit), k=val.rows(*shape, unit=unit), v=val.normal(*shape, dtype=bf16),
        gate=_cumulative(val.log_gate(*shape, decay=case["decay"]), marks), beta=val.beta(*shape[:3]), h0=None)
    if case["state"]:
        state["h0"] = val.normal(sequences or batch, heads, D, D, scale=0.02)
    if kind == "train":
        leaves = [state[n] for n in ("q", "k", "v", "gate", "beta", "h0") if state[n] is not None]
        state["leaves"] = [t.requires_grad_() for t in leaves]
        state["d_out"] = val.normal(*shape, dtype=bf16)
        if case["state"]:
            state["d_state"] = val.normal(sequences or batch, heads, D, D)
    return state


def run(state):
    case, kind = state["case"], state["case"]["kind"]
    if kind == "decode":
        with torch.no_grad():
            out = kda_b200.decode_step(state["x"], state["weight"], state["conv"], state["raw"],
                                       state["a_log"], state["bias"], state["beta"], state["pool"],
                                       state["slots"])
        return [out, state["conv"], state["pool"]]
    if kind == "extend":
        with torch.no_grad():
            out, _ = kda_b200.recurrent_kda(state["q"], state["k"], state["v"], state["gate"],
                                            state["beta"], state["pool"], cu_seqlens=state["cu"],
                                            state_indices=state["slots"])
        return [out, state["pool"]]
    if kind == "scan":
        with torch.no_grad():
            return kda_b200.chunk_kda(state["q"], state["k"], state["v"], state["gate"],
                                      state["beta"], output_final_state=True)
    if kind == "layer":
        out = state["layer"](state["x"], cu_seqlens=state["cu"]).hidden_states
        return [out, *torch.autograd.grad(out, [state["x"], *state["params"]], state["d_out"])]
    args = (state["q"], state["k"], state["v"], state["gate"], state["beta"], state["h0"])
    if kind == "prefill":
        with torch.no_grad():
            return kda_b200.chunk_kda(*args, cu_seqlens=state["cu"], output_final_state=True,
                                      normalize_qk=case["normalize"])
    out, final = kda_b200.chunk_kda(*args, cu_seqlens=state["cu"], output_final_state=case["state"],
                                    normalize_qk=case["normalize"], recompute=case["recompute"])
    outs, cotangents = ([out, final], [state["d_out"], state["d_state"]]) if case["state"] else ([out], [state["d_out"]])
    return [*outs, *torch.autograd.grad(outs, state["leaves"], cotangents)]


# flops of one (token, head) at K = V = D: forward = two gated 64-wide products, w and u, the 64-wide
# triangular inverse, the state products [w; qg] h, kg^T v_new and Aqk v_new; backward = 2.5 times
_P, _S = 2 * CHUNK * D, 2 * D * D
_FORWARD_FLOPS = 5 * _P + 3 * _S + CHUNK * CHUNK * 2 // 3
_BACKWARD_FLOPS = 11 * _P + 6 * _S


def work(case):
    kind, heads = case["kind"], case["heads"]
    if kind == "decode":
        n = case["sequences"]
        # states and histories in and out, the projections in, the row out, conv weights once
        per = 2 * 4 * D * D + (3 * 2 * 3 + 3) * 2 * D + 2 * D + 4 + 2 * D
        return {"bytes": heads * (n * per + 3 * D * 4 * 2 + 4 * D), "flops": n * heads * 7 * D * D}
    if kind == "extend":
        n, t = case["sequences"], case["tokens"]
        return {"bytes": heads * (n * 2 * 4 * D * D + t * (4 * 2 * D + 4 * D + 4)), "flops": t * heads * 7 * D * D}
    if kind == "scan":
        d, rows = case["dim"], case["batch"] * case["tokens"] * heads
        return {"bytes": rows * (5 * 4 * d + 4) + case["batch"] * heads * 4 * d * d, "flops": rows * 7 * d * d}
    units = case["batch"] * case["tokens"] * heads
    states = (case["sequences"] or case["batch"]) * heads * 4 * D * D
    forward = 4 * 2 * D + 4 * D + 4
    if kind == "prefill":
        return {"bytes": units * forward + states * (2 if case["state"] else 1), "flops": units * _FORWARD_FLOPS}
    if kind == "train":
        backward = 2 * D + 3 * 2 * D + 4 * D + 4           # dO in, gradients out
        return {"bytes": units * (forward + backward) + (4 * states if case["state"] else 0),
                "flops": units * (_FORWARD_FLOPS + _BACKWARD_FLOPS)}
    # a layer: the weights (fp32) and their gradients, hidden rows and their gradients both ways
    hidden, width, rows = case["hidden"], heads * D, case["batch"] * case["tokens"]
    weights = hidden * (4 * width + heads + 2 * D) + 2 * D * width
    return {"bytes": 2 * 4 * weights + rows * hidden * 2 * 4,
            "flops": 6 * rows * weights + units * (_FORWARD_FLOPS + _BACKWARD_FLOPS)}


def tolerance(case):
    """About four times the error against an fp32 or fp64 evaluation of the same inputs: the scan 1.6e-7
    (largest element 1.2e-6); decode 2.9e-3 (1.3e-2) and extend 1.7e-3 (4e-3), bf16 rows and outputs;
    prefill and train up to 5.2e-3 (0.12), bf16 products in several stages; layer up to 1.2e-2 in the
    gradients of the gate's parameters, 8e-3 elsewhere (0.13)."""
    kind = case["kind"]
    if kind == "scan":
        return {"rel": 1e-6, "max": 1e-5}
    if kind == "extend":
        return {"rel": 7e-3, "max": 2e-2}
    if kind == "decode":
        return {"rel": 1.2e-2, "max": 5e-2}
    return {"rel": 2.5e-2 if kind == "layer" else 2e-2, "max": 0.5}
