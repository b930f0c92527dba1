"""Gated linear attention: a recurrent mixer with one D x V float32 state matrix per head and request
(key channel x value channel), kept in the request's slot between steps.

With q = W_q x * D^(-1/2), k = W_k x (heads x D), v = W_v x (heads x V) and a decay per key channel
a = sigmoid(W_a2 (W_a1 x) + b)^(1 / tau), per head:

    S_t = diag(a_t) S_(t-1) + k_t v_t^T        o_t = S_t^T q_t

Each head's o is divided by its root mean square and multiplied by a weight over V that all heads
share; the heads, concatenated, are multiplied by silu(W_g x) and go through W_o into the stream.
The five input products run as ONE product with float32 output; decay, state and recurrence are
float32 in both engines (csrc/gla.cu).

Parameters: ``hidden_size``, ``num_heads``, ``head_dim``, ``v_dim``, ``decay_rank``, ``tau``, ``eps``.
Tensors below the prefix: q, k [H D, hidden]; v, g [H V, hidden]; a1 [rank, hidden]; a2 [H D, rank];
a2.b [H D]; norm [V]; o [hidden, H V].
"""
from __future__ import annotations

import numpy as np
import torch

from .. import ops
from ..config.spec import PartSpec
from .base import MIXERS, Mixer, StateSpec, TensorSpec
from .linear import Linear


# Tokens from which on a request's portion goes chunk by chunk in the bfloat16 engine (csrc/gla_chunked.cu): few tokens are
# through the scan before three kernels have ended (16 heads of 64 x 128, one request: 128 tokens 20 us against 33, 192 29
# against 35, 256 37 against 36, 320 46 against 35, 2,048 275 against 76), many keep all SMs at work (4 x 128: 41 against 37; 32 x
# 64: 128 against 85; but 64 x 32: 137 against 136, 128 x 16: 159 against 343).  Beside decoding requests the chunks win earlier on
# the GPU (8 of them: 128 tokens 47 against 35, 256 85 against 35), but a step of fewer than ``FEW`` tokens in chunks waits for
# the host, which launches three kernels a layer more (8 + 256 tokens at eight layers: 2.07 ms a step against 2.18).
LEAST_ALONE, LEAST_OF_MANY, FEW, MANY = 192, 64, 320, 1024


def portions_in_chunks(lengths) -> int:
    """The fewest tokens of a portion that goes chunk by chunk in a step of requests with so many (numpy integers); 0: none."""
    if lengths[lengths >= LEAST_OF_MANY].sum() >= MANY:
        return LEAST_OF_MANY
    return LEAST_ALONE if lengths[lengths >= LEAST_ALONE].sum() >= FEW else 0


@MIXERS.register("gated_linear_attention")
class GatedLinearAttention(Mixer):
    graph_safe = True  # a step of single tokens plans nothing on the host: requests and slots are read on the device

    def __init__(self, spec: PartSpec):
        super().__init__(spec)
        p = spec.params
        self.hidden_size = int(p["hidden_size"])
        self.num_heads = int(p["num_heads"])
        self.head_dim = int(p["head_dim"])
        self.v_dim = int(p["v_dim"])
        self.rank = int(p["decay_rank"])
        self.tau = float(p["tau"])
        self.eps = float(p["eps"])
        if self.head_dim > 256 or self.v_dim > 256:
            raise ValueError(f"head sizes {self.head_dim} x {self.v_dim} are not supported by the scan kernel (up to 256)")
        self.k_size = self.num_heads * self.head_dim
        self.v_size = self.num_heads * self.v_dim
        self.in_proj: Linear | None = None
        self.o_proj: Linear | None = None
        self.a2 = self.a2_bias = self.norm_weight = None

    def state_spec(self) -> StateSpec:
        return StateSpec((self.num_heads, self.head_dim, self.v_dim), "float32")

    @classmethod
    def expected_tensors(cls, spec: PartSpec, prefix: str) -> list[TensorSpec]:
        p = spec.params
        hidden, rank = int(p["hidden_size"]), int(p["decay_rank"])
        k_size, v_size = int(p["num_heads"]) * int(p["head_dim"]), int(p["num_heads"]) * int(p["v_dim"])
        return [TensorSpec(prefix + "q", (k_size, hidden)), TensorSpec(prefix + "k", (k_size, hidden)),
                TensorSpec(prefix + "v", (v_size, hidden)), TensorSpec(prefix + "g", (v_size, hidden)),
                TensorSpec(prefix + "o", (hidden, v_size)), TensorSpec(prefix + "norm", (int(p["v_dim"]),), init="ones"),
                TensorSpec(prefix + "a1", (rank, hidden)), TensorSpec(prefix + "a2", (k_size, rank)),
                TensorSpec(prefix + "a2.b", (k_size,))]

    def load(self, tensors: dict, prefix: str, device, dtype) -> None:
        fused = torch.cat([tensors[prefix + name] for name in ("q", "k", "v", "g", "a1")], dim=0)
        self.in_proj = Linear(fused, None, device, dtype)
        self.o_proj = Linear(tensors[prefix + "o"], None, device, dtype)
        f32 = lambda name: tensors[prefix + name].to(device=device, dtype=torch.float32).contiguous()
        self.a2_bias, self.norm_weight = f32("a2.b"), f32("norm")
        self.a2 = f32("a2").t().contiguous()  # [rank, H D]: the threads of a block read consecutive entries

    def _chunked(self, ctx, proj) -> tuple:
        """(chunks of the requests whose portions go chunk by chunk, the fewest tokens of one, whether other requests are in
        the step).  Only in the bfloat16 engine: the float32 engine's numbers do not depend on how a sequence is cut."""
        if (ctx.decode_only or ctx.max_q_len < LEAST_OF_MANY or ctx.dtype != torch.bfloat16 or self.head_dim > 64
                or self.head_dim % 4 or self.v_dim % 4 or proj.stride(0) % 4):
            return 0, 0, True
        plan = ctx.plans.get("gla_chunked")
        if plan is None:
            lengths = np.diff(ctx.req_indptr_host)
            least = portions_in_chunks(lengths)
            long = lengths[lengths >= least] if least else lengths[:0]
            plan = ctx.plans["gla_chunked"] = (int((-(-long // ops.gla_chunk_tokens())).sum()), least, long.size < lengths.size)
        return plan

    def forward(self, ctx, x, acc, cache) -> None:
        tokens, H, D, V = x.shape[0], self.num_heads, self.head_dim, self.v_dim
        proj = ctx.buffer("gla.proj", (tokens, 2 * self.k_size + 2 * self.v_size + self.rank), torch.float32)
        self.in_proj.forward(x, proj)
        decay = ctx.buffer("gla.decay", (tokens, self.k_size), torch.float32)
        ops.gla_decay(proj, 2 * self.k_size + 2 * self.v_size, self.a2, self.a2_bias, decay, self.rank, self.tau)
        o = ctx.buffer("gla.o", (tokens, self.v_size), torch.float32)
        chunks, least, others = self._chunked(ctx, proj)
        if others:
            ops.gla_scan(proj, decay, ctx.req_indptr, ctx.slots, cache.state, o, ctx.num_requests, H, D, V, D ** -0.5,
                         below=least if chunks else None)
        if chunks:
            # room for the chunks of any step of the token budget: portions of a chunk and a token have two chunks each
            rows = max(ctx.token_capacity, tokens)
            most = 2 * -(-rows // ops.gla_chunk_tokens())
            workspace = ctx.buffer("gla.chunks", (rows, -(-most * H * (D * V + 64) // rows)), torch.float32)
            ops.gla_chunked(proj, decay, ctx.req_indptr, ctx.slots, cache.state, o, workspace, ctx.num_requests, chunks,
                            least, H, D, V, D ** -0.5)
        out = ctx.buffer("gla.out", (tokens, self.v_size), ctx.dtype)
        ops.gla_finish(o, proj, 2 * self.k_size + self.v_size, self.norm_weight, out, H, V, self.eps)
        if not self.o_proj.accumulate_later(ctx, out, acc):
            self.o_proj.forward(out, acc, accumulate=True)
