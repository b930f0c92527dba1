"""Generalized delta rule: a recurrent mixer with one D x D float32 state matrix per head and
request (key channel x value channel), kept in the request's slot between steps.

With r, k, v = W_r x, W_k x, W_v x (heads x D each), the unit key u = k / sqrt(sum(k^2) + 1e-6),
the decay w = exp(-exp(-1/2) sigmoid(W_w2 tanh(W_w1 x) + w0)) and the removal rate
a = sigmoid(W_a x + b_a), per head and key channel:

    S_t = diag(w_t) S_(t-1) - (a_t * u_t) (u_t^T S_(t-1)) + k_t v_t^T        o_t = S_t^T r_t

Each head's o is divided by its root mean square, multiplied by a weight over all heads and by
sigmoid(W_g x), and goes through W_o into the stream.  The six input products run as ONE product
with float32 output; gates, state and recurrence are float32 in both engines (csrc/delta_rule.cu).

Parameters: ``hidden_size``, ``num_heads``, ``head_dim``, ``decay_rank``, ``eps``.  Tensors below
the prefix: r, k, v, g, a [H D, hidden]; a.b, w0, norm [H D]; w1 [rank, hidden]; w2 [H D, rank];
o [hidden, H D].
"""
from __future__ import annotations

import functools

import numpy as np
import torch

from .. import ops
from ..config.spec import PartSpec
from .base import MIXERS, Mixer, StateSpec, TensorSpec
from .linear import Linear


# Tokens from which on a request's portion goes chunk by chunk in the bfloat16 engine (csrc/delta_chunked.cu), and how many
# blocks of 16 columns an SM at most: the chunks shorten a chain that waits; where blocks enough are there to fill its waits,
# their larger preparation costs more (32 heads of 64: 1 request of 32 tokens 22 -> 18 us, of 2,048 429 -> 286; 4 of 64
# 41 -> 37, of 128 61 -> 64, of 512 236 -> 252; 32 of 64 183 -> 245).
# Beside other requests, which keep the two token-wise kernels, two kernels more have to be won back (32 heads of 64 and 8
# decoding requests: 32 tokens 33 -> 36 us, 64 44 -> 44, 96 61 -> 52, 128 77 -> 59, 512 258 -> 153), all the more where the step
# brings 64 tokens a request, since the token-wise scan of all then splits its columns (1 decoding request: 128 tokens 49 -> 58,
# 192 63 -> 66, 256 77 -> 74, 512 132 -> 119).
LEAST_CHUNKED, LEAST_BESIDE, LEAST_BESIDE_FEW, BLOCKS_AN_SM, COLUMNS = 32, 96, 256, 2, 16


def portions_in_chunks(lengths) -> int:
    """The fewest tokens of a portion that goes chunk by chunk in a step of requests with so many (numpy integers)."""
    if lengths.min() >= LEAST_CHUNKED:
        return LEAST_CHUNKED
    return LEAST_BESIDE_FEW if lengths.sum() >= 64 * lengths.size else LEAST_BESIDE


# The chunks' records: as many bytes at most (two passes over half of the chunks each: 2,048 tokens of 32 heads 292 -> 298 us; 127
# MB in one), but room for so many chunks, and for so many more than whole ones where requests end in a part of one.
RECORD_BYTES, LEAST_ROOM, PARTIAL_CHUNKS = 128 << 20, 64, 16


@functools.lru_cache(maxsize=None)
def _sm_count(device_index: int) -> int:
    return torch.cuda.get_device_properties(device_index).multi_processor_count


@MIXERS.register("general_delta")
class GeneralDeltaMixer(Mixer):
    graph_safe = True  # a step of single tokens plans nothing on the host: requests and slots are read on the device

    def __init__(self, spec: PartSpec):
        super().__init__(spec)
        p = spec.params
        self.hidden_size = int(p["hidden_size"])
        self.num_heads = int(p["num_heads"])
        self.head_dim = int(p["head_dim"])
        self.rank = int(p["decay_rank"])
        self.eps = float(p["eps"])
        if self.head_dim > 256:
            raise ValueError(f"head_dim {self.head_dim} is not supported by the delta-rule kernels (up to 256)")
        self.size = self.num_heads * self.head_dim
        self.in_proj: Linear | None = None
        self.o_proj: Linear | None = None
        self.w2 = self.w0 = self.a_bias = self.norm_weight = None

    def state_spec(self) -> StateSpec:
        return StateSpec((self.num_heads, self.head_dim, self.head_dim), "float32")

    @classmethod
    def expected_tensors(cls, spec: PartSpec, prefix: str) -> list[TensorSpec]:
        p = spec.params
        hidden, size, rank = int(p["hidden_size"]), int(p["num_heads"]) * int(p["head_dim"]), int(p["decay_rank"])
        out = [TensorSpec(prefix + name, (size, hidden)) for name in ("r", "k", "v", "g", "a")]
        out += [TensorSpec(prefix + "a.b", (size,)), TensorSpec(prefix + "w1", (rank, hidden)),
                TensorSpec(prefix + "w2", (size, rank)), TensorSpec(prefix + "w0", (size,)),
                TensorSpec(prefix + "norm", (size,), init="ones"), TensorSpec(prefix + "o", (hidden, size))]
        return out

    def load(self, tensors: dict, prefix: str, device, dtype) -> None:
        fused = torch.cat([tensors[prefix + name] for name in ("r", "k", "v", "g", "a", "w1")], dim=0)
        self.in_proj = Linear(fused, None, device, dtype)
        self.o_proj = Linear(tensors[prefix + "o"], None, device, dtype)
        f32 = lambda name: tensors[prefix + name].to(device=device, dtype=torch.float32).contiguous()
        self.w0, self.a_bias, self.norm_weight = f32("w0"), f32("a.b"), f32("norm")
        self.w2 = f32("w2").t().contiguous()  # [rank, H D]: the threads of a block read consecutive entries

    def _scratch_rows(self, rows: int, chunked: bool) -> tuple:
        """(rows of the scratch memory of an engine whose steps bring up to ``rows`` tokens, chunks it has room for).  It holds the
        gates, [tokens, H 3 D], and in their turn the records of a step's chunks (2.4 times the gates at D 64), but no more than
        ``RECORD_BYTES`` of them: a step of more chunks goes in passes.  The size does not depend on the step, so the first one
        allocates it for good."""
        if not chunked:
            return rows, 0
        record = self.num_heads * ops.delta_chunk_record()
        room = -(-rows // ops.delta_chunk_tokens()) + PARTIAL_CHUNKS
        room = max(LEAST_ROOM, min(room, RECORD_BYTES // (4 * record)))
        return max(rows, -(-room * record // (3 * self.size))), room

    def _plan(self, ctx, tokens: int) -> tuple:
        """(scratch memory, its rows for the gates, the passes of the requests whose portions go chunk by chunk, their chunks and
        fewest tokens, whether other requests are in the step), the same for every such layer of a step.  Chunks only in the bfloat16 engine: the
        float32 engine's numbers do not depend on how a sequence is cut."""
        key = ("delta_rule", self.num_heads, self.head_dim)
        plan = ctx.plans.get(key)
        if plan is None:
            chunked = ctx.dtype == torch.bfloat16 and self.head_dim <= 64 and self.head_dim % 4 == 0
            rows, room = self._scratch_rows(max(ctx.token_capacity, tokens), chunked)
            work = ctx.buffer(f"delta.work{self.head_dim}", (rows, 3 * self.size), torch.float32)
            passes, chunks, least, others = None, 0, 0, True
            if chunked and not ctx.decode_only and ctx.max_q_len >= LEAST_CHUNKED:
                lengths = np.diff(ctx.req_indptr_host)
                least = portions_in_chunks(lengths)
                long = lengths[lengths >= least]
                blocks = long.size * self.num_heads * -(-self.head_dim // COLUMNS)
                if 0 < long.size <= room and blocks <= BLOCKS_AN_SM * _sm_count(torch.cuda.current_device()):
                    each = -(-long // ops.delta_chunk_tokens())
                    passes, chunks, others = ops.delta_chunk_passes(each, room), int(each.sum()), long.size < lengths.size
            plan = ctx.plans[key] = (work, work[:tokens], passes, chunks, least, others)
        return plan

    def forward(self, ctx, x, acc, cache) -> None:
        tokens, H, D = x.shape[0], self.num_heads, self.head_dim
        proj = ctx.buffer("delta.proj", (tokens, 5 * self.size + self.rank), torch.float32)
        self.in_proj.forward(x, proj)
        o = ctx.buffer("delta.o", (tokens, self.size), torch.float32)
        work, gates, passes, chunks, least, others = self._plan(ctx, tokens)
        if others:
            ops.delta_prepare(proj, self.w2, self.w0, self.a_bias, gates, H, D, self.rank)
            ops.delta_scan(proj, gates, ctx.req_indptr, ctx.slots, cache.state, o, ctx.num_requests, H, D,
                           below=least if chunks else None)
        if chunks:  # their records take the place of the gates, which nothing reads any more
            ops.delta_chunked(proj, self.w2, self.w0, self.a_bias, ctx.req_indptr, ctx.slots, cache.state, o, work,
                              ctx.num_requests, chunks, least, H, D, self.rank, passes)
        out = ctx.buffer("delta.out", (tokens, self.size), ctx.dtype)
        ops.delta_finish(o, proj, self.norm_weight, out, H, D, self.eps)
        if not self.o_proj.accumulate_later(ctx, out, acc):
            self.o_proj.forward(out, acc, accumulate=True)
