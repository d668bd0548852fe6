"""Linear attention with a constant decay per head ("lightning attention").

With mixer input h, H heads, key size dk and value size dv:
    q = act(W_q h), k = act(W_k h)  [H, dk],   v = act(W_v h)  [H, dv]        act = silu
    S_h <- decay_h * S_h + k_h v_h^T ,   o_h = S_h^T q_h                       per head, token by token
    out = W_o ( rmsnorm(o over all heads) * w * sigmoid(W_g h) )
A request's state is S [H, dk, dv] in 32 bit, zero at its start, one per run of the layer; a step continues from what
the request's earlier steps left, so a prompt may be cut anywhere.  The four projections are one product; the
recurrence, its decays and the norm are 32 bit whatever the compute type.  Steps of single tokens stream the state through
registers once; short portions run one block per (row, head) over the row's chunks in turn; long portions run their chunks in parallel (``csrc/decay_attention.cu``;
heads of 64 or 128 entries in chunks of 64 tokens where those are enough blocks, ``csrc/decay_attention_tiles.cu``; heads of 128 x 128 in chunks of 128 on the
tensor cores where those are full enough, ``csrc/decay_attention_tc.cu``).
"""
from __future__ import annotations

import torch

from ..kernels import ops
from . import linear
from .base import MIXERS, Mixer, StateSpec, TensorSpec
from .chunks import chunk_layout

STATE = "decay_attention"
PARALLEL_FROM = 65      # portions of at least this many tokens run their chunks in parallel


def tiles_pay(q_lens, chunk: int, heads: int, sm_count: int) -> bool:
    """Whether chunks of 64 tokens give the device enough blocks (one a chunk and head): a block works twice as long as one of the kernels with
    chunks of 32.  The layer of 8 heads (16 heads), microseconds, chunks of 64 against 32: 65 tokens, 16 (32) blocks, 69 against 60 (77, 68);
    257 tokens, 40 (80) blocks, 71 against 61 (81, 81); 500 tokens, 64 (128) blocks, 76 against 72 (88, 116); eight rows of 65 76 against 107."""
    return 2 * heads * sum(-(-n // chunk) for n in q_lens) >= sm_count


def tensor_cores_pay(q_lens, chunk: int, heads: int, sm_count: int) -> bool:
    """Whether a step's portions (heads of 128 x 128, bfloat16) go to the tcgen05 kernels with chunks of 128 tokens or to the FMA kernels in chunks of 64
    and 32.  A block of the former holds an SM alone, full chunk or single token.  Where all run at once they are ahead in the layer, with its launches and products
    beside them (microseconds, tcgen05 and FMA): 8 heads, 65 tokens 103, 109; two rows of 150 99, 106; 65 beside 16 single ones 112, 121; 16 heads, 300 beside
    four of 20 101, 105.  Then every time that the SMs have one each takes about 47, and the others' time follows tokens and chunks of 64.  The kernels alone, everything cold,
    16 heads: eight rows of 65 tokens 73, 87; four of 500 108, 163; 20 of 100 165, 200; 65 tokens beside 16 / 32 single ones 120 / 220, 77 / 110; 2,000 beside 32 single ones
    382, 304; 300 beside 16 of 20 159, 103.  32 heads: 15 rows of 130 343, 380; 512 tokens beside 8 single ones 169, 134."""
    blocks = heads * sum([-(-n // chunk) for n in q_lens])
    if blocks <= sm_count:
        return True
    halves = heads * sum([-(-n // (chunk // 2)) for n in q_lens])
    return 20 + 47 * -(-blocks // sm_count) <= 40 + (0.27 * heads * sum(q_lens) + 21 * halves) / sm_count


@MIXERS.register("decay_attention")
class DecayAttention(Mixer):
    """Tensor names under ``prefix``: ``q``, ``k`` [H*dk, d], ``v``, ``g`` [H*dv, d], ``norm`` [H*dv], ``o`` [d, H*dv]."""

    def __init__(self, prefix: str, width: int, heads: int, head_dim: int, value_dim: int, decays, eps: float):
        self.prefix, self.width = prefix, int(width)
        self.heads, self.dk, self.dv = int(heads), int(head_dim), int(value_dim)
        self.decays = [float(x) for x in decays]
        if len(self.decays) != self.heads:
            raise ValueError(f"{len(self.decays)} decays for {self.heads} heads")
        self.eps = float(eps)
        self.w_in = self.w_o = self.norm_w = self._decays = None
        self._most = (None, 0)      # the engine's limits, and the most floats that a step's chunks take under them

    def tensor_specs(self):
        p, d, H, dk, dv = self.prefix, self.width, self.heads, self.dk, self.dv
        return [TensorSpec(p + "q", (H * dk, d)), TensorSpec(p + "k", (H * dk, d)), TensorSpec(p + "v", (H * dv, d)),
                TensorSpec(p + "g", (H * dv, d)), TensorSpec(p + "norm", (H * dv,), kind="vector", init="norm"),
                TensorSpec(p + "o", (d, H * dv))]

    def bind(self, tensors):
        p = self.prefix
        self.w_in = torch.cat([tensors[p + "q"], tensors[p + "k"], tensors[p + "v"], tensors[p + "g"]], dim=0).contiguous()
        self.w_o = tensors[p + "o"]
        self.norm_w = tensors[p + "norm"].float().contiguous()
        self._decays = torch.tensor(self.decays, dtype=torch.float64, device=self.w_o.device)

    def run_state_specs(self):
        return {STATE: StateSpec((self.heads, self.dk, self.dv), torch.float32, 0.0)}

    def _chunks(self, ctx, floats: int, tensor_cores: bool):
        """Working memory for a step's chunks: one buffer, whichever of the forms that these heads have a step takes (chunks of 64, and of 128 on the tensor cores
        or of 32)."""
        key = (ctx.max_step_tokens, ctx.max_rows, tensor_cores)
        if self._most[0] != key:      # (the host's time counts in short steps)
            forms = [(ops.decay_attention_tc_chunk() if tensor_cores else ops.decay_attention_chunk(), self.dk * self.dv)]
            if ops.decay_attention_tiles_supported(self.dk, self.dv, 8, 0, 0, 0):
                forms.append((ops.decay_attention_tiles_chunk(), ops.decay_attention_tiles_floats(self.dk, self.dv)))
            self._most = (key, self.heads * max((-(-key[0] // chunk) + key[1]) * per for chunk, per in forms))
        return ctx.scratch("decay_attention.chunks", (floats,), torch.float32, bound=(self._most[1],))

    def forward(self, ctx, x, cache):
        H, dk, dv = self.heads, self.dk, self.dv
        T = x.shape[0]
        qkvg = linear.linear(ctx, x, self.w_in)                       # [T, 2 H dk + 2 H dv]: q | k | v | g, before activations
        o = torch.empty((T, H * dv), dtype=torch.float32, device=x.device)
        rows = dict(row_slot=ctx.row_slot, row_q_start=ctx.row_q_start, row_q_len=ctx.row_q_len)
        portions = not ctx.replayable and ctx.max_q_len >= PARALLEL_FROM
        # long portions: the recurrence is linear in the state, so a row's chunks run in parallel and are stitched together
        tc = portions and ops.decay_attention_tc_supported(dk, dv, qkvg.shape[1], 0, H * dk, 2 * H * dk, x.dtype)
        long = ops.decay_attention_tc_chunk() if tc else 0
        if tc and tensor_cores_pay(ctx.host["q_lens"], long, H, ctx.sm_count):
            base, total, most = chunk_layout(ctx, long)
            work = self._chunks(ctx, total * H * dk * dv, tc)
            ops.decay_attention_tc(qkvg, 0, H * dk, 2 * H * dk, self._decays, cache.state[STATE], o, work, base, most, H=H, dk=dk, dv=dv, silu=True,
                                   err=ctx.err, **rows)
        elif (portions and ops.decay_attention_tiles_supported(dk, dv, qkvg.shape[1], 0, H * dk, 2 * H * dk)
                and tiles_pay(ctx.host["q_lens"], ops.decay_attention_tiles_chunk(), H, ctx.sm_count)):
            base, total, most = chunk_layout(ctx, ops.decay_attention_tiles_chunk())
            work = self._chunks(ctx, total * H * ops.decay_attention_tiles_floats(dk, dv), tc)
            ops.decay_attention_tiles(qkvg, 0, H * dk, 2 * H * dk, self._decays, cache.state[STATE], o, work, base, total, most, H=H, dk=dk,
                                      dv=dv, silu=True, **rows)
        elif portions and ops.decay_attention_chunked_supported(dk, dv):
            chunk = ops.decay_attention_chunk()

            def layout():
                counts = [-(-n // chunk) for n in ctx.host["q_lens"]]
                base = [sum(counts[:i]) for i in range(len(counts))]
                return torch.tensor(base, dtype=torch.int32).to(x.device, non_blocking=True), sum(counts), max(counts)
            base, total, most = ctx.memo(("decay_attention chunks", chunk), layout)
            work = self._chunks(ctx, total * H * dk * dv, tc)
            ops.decay_attention_chunked(qkvg, 0, H * dk, 2 * H * dk, self._decays, cache.state[STATE], o, work, base, most, H=H, dk=dk,
                                        dv=dv, silu=True, **rows)
        elif ctx.decode_only and ops.decay_attention_step_supported(dk, dv):
            ops.decay_attention_step(qkvg, 0, H * dk, 2 * H * dk, self._decays, cache.state[STATE], o, H=H, dk=dk, dv=dv, silu=True,
                                     row_slot=ctx.row_slot, row_q_start=ctx.row_q_start)
        else:
            ops.decay_attention(qkvg, 0, H * dk, 2 * H * dk, self._decays, cache.state[STATE], o, H=H, dk=dk, dv=dv, silu=True, **rows)
        y = torch.empty((T, H * dv), dtype=x.dtype, device=x.device)
        g_at = qkvg.data_ptr() + (2 * H * dk + H * dv) * qkvg.element_size()
        ops.gated_rms_norm(o, g_at, qkvg.shape[1], self.norm_w, y, self.eps)
        return linear.linear(ctx, y, self.w_o)
