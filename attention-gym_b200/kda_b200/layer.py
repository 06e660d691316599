"""``KDAAttention``: the trainable KDA layer assembled from this package's kernels.

Same module interface as the reference's example layer (examples/kda_training.py:151-538):
constructor arguments, parameter names and shapes, the ``forward`` signature and the
``KDAAttentionOutput`` result, so a checkpoint or a caller of that module fits this one.  Data
flow of ``forward`` (reference lines in brackets):

    hidden --qkv_proj--> qkv --causal_conv1d + SiLU--> q | k | v           [:358-410]
    q, k --l2norm--> unit rows                                             [:412-421]
    hidden --f_a_proj, f_b_proj--> raw gate;  hidden --beta_proj, sigmoid--> beta   [:423-446]
    raw gate --bounded_gate_cumsum--> cumulative log2 gate                 [:448-475]
    chunk_kda(q, k, v, gate, beta) --> o, final state                      [:477-505]
    o, g_b_proj(g_a_proj(hidden)) --gated_output_norm--> y --out_proj--> result    [:507-539]

The projections are cuBLAS GEMMs (``F.linear``); everything between them is this package:
one conv kernel, one gate kernel, the chunked core with the q / k L2 normalisation fused into its
first forward and last backward kernel (``fuse_qk_norm=False`` runs the two l2norm launches of the
reference instead), and the output epilogue ``rms_norm(o) * weight * sigmoid(gate logits)`` as ONE
kernel where the reference runs three.
Packed inputs share one chunk schedule between the gate and the core, as in the reference.
``backend="reference"`` evaluates the same layer in eager fp32 PyTorch (dense inputs only), for
parity checks; there is no fallback from one backend to the other.
"""

from __future__ import annotations

import math
from typing import NamedTuple, Optional

import torch
import torch.nn as nn
import torch.nn.functional as F

from .chunk_schedule import prepare_ragged_chunk_metadata
from .fused import chunk_forward as _chunk_kda, chunk_forward_qkv as _chunk_kda_qkv
from .masking import active_token_mask, mask_inactive_token_gradients, mask_inactive_tokens
from .ops import widen_op
from .preops import _bounded_gate_cumsum, causal_conv1d, gated_output_norm, l2norm
from .reference_impl import reference_kda

_LOG2E = math.log2(math.e)


# Elements from which _CastWeight's gain of 1.84 us a million outweighs the 14 us of host that it costs forward and backward (without
# this line it was 4 to 7 % of a step of layers with 512 to 1024 channels).  Not an attribute of the class: a full-graph trace
# cannot compare with those.
_WIDEN_ELEMENTS = 2 ** 23


class _CastWeight(torch.autograd.Function):
    """``weight.to(torch.bfloat16)`` of a large fp32 parameter (fused backend); the same values both ways.  The gradient goes
    back to fp32 in a streaming kernel: 50 M elements take 46 us, the copy kernel behind ``.to`` 138."""

    @staticmethod
    def forward(ctx, weight):
        return weight.to(torch.bfloat16)

    @staticmethod
    def backward(ctx, grad):
        if torch.is_grad_enabled():            # to be differentiated once more
            return grad.to(torch.float32)
        return widen_op(grad)


class KDAAttentionOutput(NamedTuple):
    """Hidden states and optional recurrent and convolution states."""

    hidden_states: torch.Tensor
    final_state: Optional[torch.Tensor]
    final_conv_state: Optional[torch.Tensor]


class KDAAttention(nn.Module):
    """KDA attention layer.  ``mask_inactive_capacity=True`` makes a packed input whose buffer is
    longer than ``cu_seqlens[-1]`` safe for training: the rows past the end are zeroed on the way in
    and kept out of every weight gradient (the primitives leave them undefined)."""

    def __init__(self, hidden_size: int, num_heads: int, head_dim: int, *, chunk_size: int = 64,
                 short_conv_kernel_size: int = 4, lower_bound: float = -5.0,
                 backend: str = "fused", fastmath: bool = False, rms_norm_eps: float = 1e-5,
                 compute_dtype: Optional[torch.dtype] = None, device=None,
                 mask_inactive_capacity: bool = False, fuse_qk_norm: bool = True) -> None:
        super().__init__()
        if hidden_size < 1 or num_heads < 1 or head_dim < 1:
            raise ValueError("hidden_size, num_heads, and head_dim must be positive")
        if chunk_size < 1:
            raise ValueError(f"chunk_size must be positive, got {chunk_size}")
        if short_conv_kernel_size < 1:
            raise ValueError(f"short_conv_kernel_size must be positive, got {short_conv_kernel_size}")
        if not math.isfinite(lower_bound) or lower_bound > 0:
            raise ValueError(f"lower_bound must be finite and non-positive, got {lower_bound}")
        if backend not in ("reference", "fused"):
            raise ValueError(f"backend must be 'reference' or 'fused', got {backend!r}")
        if backend == "fused" and (head_dim != 128 or chunk_size != 64):
            raise ValueError("the fused backend requires head_dim=128 and chunk_size=64")
        self.hidden_size, self.num_heads, self.head_dim = hidden_size, num_heads, head_dim
        self.chunk_size, self.lower_bound, self.backend = chunk_size, lower_bound, backend
        self.fastmath, self.rms_norm_eps = fastmath, rms_norm_eps
        self.mask_inactive_capacity = mask_inactive_capacity
        self.fuse_qk_norm = fuse_qk_norm
        self.compute_dtype = ((torch.bfloat16 if backend == "fused" else torch.float32)
                              if compute_dtype is None else compute_dtype)
        if backend == "fused" and self.compute_dtype != torch.bfloat16:
            raise ValueError("the fused backend requires compute_dtype=torch.bfloat16")
        width = num_heads * head_dim
        kw = {"device": device}
        self.qkv_proj = nn.Linear(hidden_size, 3 * width, bias=False, **kw)
        self.qkv_conv1d = nn.Conv1d(3 * width, 3 * width, short_conv_kernel_size, groups=3 * width,
                                    bias=False, **kw)
        self.beta_proj = nn.Linear(hidden_size, num_heads, bias=False, **kw)
        self.f_a_proj = nn.Linear(hidden_size, head_dim, bias=False, **kw)
        self.f_b_proj = nn.Linear(head_dim, width, bias=False, **kw)
        self.g_a_proj = nn.Linear(hidden_size, head_dim, bias=False, **kw)
        self.g_b_proj = nn.Linear(head_dim, width, bias=False, **kw)
        self.output_norm_weight = nn.Parameter(torch.ones(head_dim, device=device, dtype=torch.float32))
        self.out_proj = nn.Linear(width, hidden_size, bias=False, **kw)
        self.A_log = nn.Parameter(torch.zeros(num_heads, device=device, dtype=torch.float32))
        self.dt_bias = nn.Parameter(torch.zeros(num_heads, head_dim, device=device, dtype=torch.float32))

    # ---- stages -------------------------------------------------------------------------------
    def _cast(self, layer):
        weight = layer.weight
        if (self.backend == "fused" and type(weight) is nn.Parameter and weight.is_cuda and weight.requires_grad
                and weight.numel() >= _WIDEN_ELEMENTS and weight.dtype == torch.float32 and torch.is_grad_enabled()):
            return _CastWeight.apply(weight)
        return weight.to(self.compute_dtype)

    def _linear(self, x, layer):
        return F.linear(x, self._cast(layer))

    def short_convolution(self, qkv, initial_state, *, cu_seqlens=None, return_final_state=False):
        batch, tokens, channels = qkv.shape
        hist = self.qkv_conv1d.kernel_size[0] - 1
        nseq = batch if cu_seqlens is None else cu_seqlens.shape[0] - 1
        if initial_state is not None:
            if tuple(initial_state.shape) != (nseq, hist, channels):
                raise ValueError(f"initial_conv_state must have shape {(nseq, hist, channels)}, "
                                 f"got {tuple(initial_state.shape)}")
            initial_state = initial_state.to(device=qkv.device, dtype=qkv.dtype).contiguous()
        weight = self.qkv_conv1d.weight[:, 0].to(self.compute_dtype)
        if self.backend == "fused":
            result = causal_conv1d(qkv, weight, activation="silu", initial_state=initial_state,
                                   cu_seqlens=cu_seqlens, return_final_state=return_final_state)
            return result if return_final_state else (result, None)
        if initial_state is None:
            initial_state = qkv.new_zeros(nseq, hist, channels)
        ext = torch.cat((initial_state, qkv), 1)
        out = F.silu(F.conv1d(ext.transpose(1, 2), self.qkv_conv1d.weight.to(self.compute_dtype),
                              groups=channels).transpose(1, 2))
        return out, (ext[:, tokens:].clone() if return_final_state else None)

    def gate_projections(self, hidden):
        return self._gates(self._linear(hidden, self.f_a_proj), self._linear(hidden, self.beta_proj))

    def _gates(self, low, beta_logits):
        batch, tokens, _ = low.shape
        raw = self._linear(low, self.f_b_proj)
        beta = beta_logits.view(batch, tokens, self.num_heads).float().sigmoid()
        return raw.view(batch, tokens, self.num_heads, self.head_dim).contiguous(), beta

    def _narrow_projections(self, hidden):
        """``f_a_proj``, ``g_a_proj`` and ``beta_proj`` in one GEMM, or None.  Each of the three reads all of ``hidden`` for 128 columns
        or fewer, forward and backward, and their input gradients have to be added.  8192 tokens of 4096 channels, us apart /
        together: forward 61 / 24, weight gradients 54 / 23, input gradients 45 / 21, their sum 93 / 30; for that two small copies of
        the weights and of the gradients, 10.  Only where the columns of every part start on 16 bytes, the weights are plain
        tensors (not sharded or quantised ones, which may not concatenate) and the class's own methods do the projections."""
        parts = (self.f_a_proj, self.g_a_proj, self.beta_proj)
        own = all(getattr(type(self), name) is method and name not in self.__dict__ for name, method in _PROJECTIONS.items())
        plain = all(type(p.weight) in (nn.Parameter, torch.Tensor) for p in parts)
        if self.backend != "fused" or not own or not plain or any(p.weight.shape[0] % 8 for p in parts):
            return None
        weights = [self._cast(p) for p in parts]
        return F.linear(hidden, torch.cat(weights)).split([w.shape[0] for w in weights], -1)

    def _reference_core(self, q, k, v, raw_gate, beta, initial_state, return_final_state):
        """Eager fp32 evaluation of the normalisation, the gate and the recurrence (dense input)."""
        q, k, v = q.float(), k.float(), v.float()
        q = q * torch.rsqrt((q * q).sum(-1, keepdim=True) + 1e-6)
        k = k * torch.rsqrt((k * k).sum(-1, keepdim=True) + 1e-6)
        z = raw_gate.float() + self.dt_bias
        gate = self.lower_bound * torch.sigmoid(self.A_log.exp().view(1, 1, -1, 1) * z) * _LOG2E
        batch, tokens = gate.shape[:2]
        pad = (-tokens) % self.chunk_size
        cum = F.pad(gate, (0, 0, 0, 0, 0, pad)).view(batch, -1, self.chunk_size, *gate.shape[2:])
        cum = cum.cumsum(2).view(batch, -1, *gate.shape[2:])[:, :tokens]
        return reference_kda("chunk", q, k, v, cum, beta, initial_state, None, return_final_state)

    # ---- forward ------------------------------------------------------------------------------
    def forward(self, hidden_states, initial_state=None, *, initial_conv_state=None, cu_seqlens=None,
                return_final_state: bool = False) -> KDAAttentionOutput:
        """hidden_states ``[B, T, hidden]`` (packed: ``[1, T, hidden]`` with ``cu_seqlens``);
        ``initial_state [N, H, D, D]``; ``initial_conv_state [N, W - 1, 3 H D]``."""
        if hidden_states.ndim != 3 or hidden_states.shape[-1] != self.hidden_size:
            raise ValueError(f"hidden_states must have shape [B, T, {self.hidden_size}], "
                             f"got {tuple(hidden_states.shape)}")
        batch, tokens, _ = hidden_states.shape
        if batch == 0 or tokens == 0:
            raise ValueError("batch size and sequence length must be greater than zero")
        if cu_seqlens is not None and self.backend != "fused":
            raise ValueError("packed cu_seqlens currently require backend='fused'")
        nseq = batch if cu_seqlens is None else cu_seqlens.shape[0] - 1
        if initial_state is not None:
            expect = (nseq, self.num_heads, self.head_dim, self.head_dim)
            if tuple(initial_state.shape) != expect:
                raise ValueError(f"initial_state must have shape {expect}, got {tuple(initial_state.shape)}")
            initial_state = initial_state.to(device=hidden_states.device, dtype=torch.float32)
        mask = (active_token_mask(hidden_states, cu_seqlens)
                if self.mask_inactive_capacity and cu_seqlens is not None else None)
        hidden = mask_inactive_tokens(hidden_states, mask).to(self.compute_dtype)
        qkv = mask_inactive_token_gradients(self._linear(hidden, self.qkv_proj), mask)
        qkv, final_conv_state = self.short_convolution(qkv, initial_conv_state, cu_seqlens=cu_seqlens,
                                                       return_final_state=return_final_state)
        qkv = mask_inactive_tokens(qkv, mask)
        qkv = qkv.view(batch, tokens, 3, self.num_heads, self.head_dim)
        narrow = self._narrow_projections(hidden)
        raw_gate, beta = self.gate_projections(hidden) if narrow is None else self._gates(narrow[0], narrow[2])
        raw_gate = mask_inactive_token_gradients(raw_gate, mask)
        beta = mask_inactive_token_gradients(beta, mask)
        if self.backend == "reference":
            out, final_state = self._reference_core(*qkv.unbind(2), raw_gate, beta, initial_state,
                                                    return_final_state)
        else:
            metadata = (None if cu_seqlens is None
                        else prepare_ragged_chunk_metadata(cu_seqlens, tokens, self.chunk_size))
            gate = _bounded_gate_cumsum(raw_gate, self.A_log, self.dt_bias, chunk_size=self.chunk_size,
                                        lower_bound=self.lower_bound, fastmath=self.fastmath,
                                        metadata=metadata)
            if self.fuse_qk_norm and qkv.dtype == torch.bfloat16:      # (what the class's own convolution returns)
                out, final_state = _chunk_kda_qkv(qkv, gate, beta, initial_state, metadata=metadata,
                                                  output_final_state=return_final_state)
            else:
                q, k, v = qkv.unbind(2)
                if not self.fuse_qk_norm:
                    q, k = l2norm(q.contiguous()), l2norm(k.contiguous())
                out, final_state = _chunk_kda(q, k, v.contiguous(), gate, beta, initial_state,
                                              metadata=metadata, output_final_state=return_final_state,
                                              fastmath=self.fastmath, normalize_qk=self.fuse_qk_norm)
        out = mask_inactive_tokens(out, mask)
        low = self._linear(hidden, self.g_a_proj) if narrow is None else narrow[1]
        logits = self._linear(low, self.g_b_proj).view_as(out)
        if self.backend == "fused":
            gated = gated_output_norm(out, logits, self.output_norm_weight, self.rms_norm_eps)
        else:
            gated = F.rms_norm(out.float(), (self.head_dim,), self.output_norm_weight,
                               eps=self.rms_norm_eps) * logits.float().sigmoid()
        result = self._linear(gated.flatten(-2).to(self.compute_dtype), self.out_proj)
        result = mask_inactive_token_gradients(result, mask)
        return KDAAttentionOutput(result.to(hidden_states.dtype), final_state, final_conv_state)


# replaced ones, in a subclass or on an object, are called for every projection (compared on the class, which a trace can do too)
_PROJECTIONS = {name: getattr(KDAAttention, name) for name in ("gate_projections", "_linear", "_cast")}

__all__ = ["KDAAttention", "KDAAttentionOutput"]
