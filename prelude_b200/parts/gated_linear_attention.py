"""Linear attention with a matrix state per head and a learned decay per key channel (``GatedLinearAttentionSpec``).

One merged projection [v | k | q | gate | narrow part of the decay].  A step of single tokens (a decode step) runs decay,
recurrence, norm per head and gate in one kernel; a step with prompt tokens makes the decays of all its tokens, runs the
recurrence over every sequence's tokens in order, then norms and gates.  The decay, its logarithm and everything of the
recurrence are float32; the state [heads, head_dim, value_dim] (float32) lives in the sequence's state slot.  The kernels
find a step's sequences through the step's device arrays, so the mixer can be recorded.
"""
from __future__ import annotations

from typing import Dict

import torch

from ..config.spec import GatedLinearAttentionSpec
from ..ops import kernels as K
from ..ops.linear import PendingProduct, linear
from ..weights.loader import ANY, TensorReq
from .registry import RunContext, StateNeed, register_part


@register_part("mixer", "gated_linear_attention")
class GatedLinearAttention:
    defer_output = False        # True: the output projection is handed on as a product still to run (``PendingProduct``)

    def __init__(self, spec: GatedLinearAttentionSpec, prefix: str):
        self.spec, self.prefix = spec, prefix
        self.qk_cols = spec.num_heads * spec.head_dim
        self.v_cols = spec.num_heads * spec.value_dim
        self.scale = float(spec.head_dim) ** -0.5
        self.w_in = self.w_a2 = self.w_o = self.a2_bias = self.norm_w = self.norm_heads = None
        self.rank = 0

    def tensors(self) -> Dict[str, TensorReq]:
        s, p = self.spec, self.prefix
        rank = ANY if s.decay_rank is None else s.decay_rank
        return {
            f"{p}.{s.q_name}": TensorReq((self.qk_cols, s.hidden_size)),
            f"{p}.{s.k_name}": TensorReq((self.qk_cols, s.hidden_size)),
            f"{p}.{s.v_name}": TensorReq((self.v_cols, s.hidden_size)),
            f"{p}.{s.gate_name}": TensorReq((self.v_cols, s.hidden_size)),
            f"{p}.{s.a1_name}": TensorReq((rank, s.hidden_size)),
            f"{p}.{s.a2_name}": TensorReq((self.qk_cols, rank)),
            f"{p}.{s.a2_name}{s.bias_suffix}": TensorReq((self.qk_cols,), "bias"),
            f"{p}.{s.norm_name}": TensorReq((s.value_dim,), "norm"),
            f"{p}.{s.o_name}": TensorReq((s.hidden_size, self.v_cols)),
        }

    def load(self, get, ctx: RunContext) -> None:
        s, p = self.spec, self.prefix

        def mat(name):
            return get(f"{p}.{name}").to(device=ctx.device, dtype=ctx.dtype)

        def vec(name):
            return get(f"{p}.{name}").to(device=ctx.device, dtype=torch.float32).contiguous()

        mats = [mat(s.v_name), mat(s.k_name), mat(s.q_name), mat(s.gate_name), mat(s.a1_name)]
        self.rank = mats[-1].shape[0]
        pad = (-sum(m.shape[0] for m in mats)) % 8             # rows of the merged projection stay 16-byte aligned
        if pad:
            mats.append(torch.zeros((pad, s.hidden_size), dtype=ctx.dtype, device=ctx.device))
        self.w_in = torch.cat(mats, dim=0).contiguous()
        self.w_a2, self.w_o = mat(s.a2_name).contiguous(), mat(s.o_name).contiguous()
        if self.w_a2.shape[1] != self.rank:
            raise ValueError(f"{p}: the decay's matrices meet at {self.rank} and {self.w_a2.shape[1]} channels")
        self.a2_bias = vec(s.a2_name + s.bias_suffix)
        self.norm_w = vec(s.norm_name)
        self.norm_heads = self.norm_w.repeat(s.num_heads).contiguous()     # one weight over value_dim, shared by the heads

    def activation_bytes_per_token(self, elem: int) -> int:
        # the scan by sixteen tokens leaves up to 26 KB a sixteen and head between its two kernels
        return ((2 * self.qk_cols + 3 * self.v_cols + self.rank + 8) * elem + (self.qk_cols + self.v_cols) * 4 + self.spec.hidden_size * elem
                + self.spec.num_heads * 1664)

    def activation_bytes_per_sequence(self) -> int:
        return self.spec.num_heads * 26624

    def cache_need(self) -> StateNeed:
        s = self.spec
        return StateNeed((s.num_heads, s.head_dim, s.value_dim), torch.float32)

    def forward(self, x: torch.Tensor, batch, cache, write_cache: bool = True):
        s = self.spec
        T = batch.n_tokens
        proj = linear(x, self.w_in)
        k0, q0 = self.v_cols, self.v_cols + self.qk_cols
        g0 = q0 + self.qk_cols
        a0 = g0 + self.v_cols
        v, k, q, gate, a1 = proj[:, :k0], proj[:, k0:q0], proj[:, q0:g0], proj[:, g0:a0], proj[:, a0:a0 + self.rank]
        y = batch.workspace("gla_gated", (T, self.v_cols), x.dtype)
        if batch.decode_only and K.gla_step_takes(cache.state):
            K.gla_step(q, k, v, a1, gate, self.w_a2, self.a2_bias, s.tau, self.scale, self.norm_w, s.norm_eps, cache.state, batch, out=y)
        else:
            decay = K.channel_decay(a1, self.w_a2, self.a2_bias, s.tau, out=batch.workspace("gla_decay", (T, self.qk_cols), torch.float32))
            o = K.gla_scan(q, k, v, decay, self.scale, cache.state, batch, out=batch.workspace("gla_o", (T, self.v_cols), torch.float32))
            K.gated_group_rmsnorm(o, gate, self.norm_heads, s.num_heads, s.norm_eps, out=y, gate_after=True)
        return PendingProduct(y, self.w_o) if self.defer_output else linear(y, self.w_o)
