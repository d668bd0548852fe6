"""The work by which the engine's speed is measured: layers at the sizes of the benchmark's models, each called as the model calls it,
and two whole steps of a Yi model that return logits.

A layer is a registered part (``delta_b200.parts``) with random weights, called with a step's context and its cache.  Prompt portions run
eagerly, with a context of their own for every pass, as in a step; single tokens run from a CUDA graph, as the engine runs decode steps.
Recurrent states are cleared at the start of a pass, as they are when a request is admitted.
"""
import math
import zlib

import numpy as np
import torch

from delta_b200.cache.manager import CacheManager
from delta_b200.config import EngineConfig
from delta_b200.engine.context import StepContext
from delta_b200.engine.step import ModelRunner, RowInput
from delta_b200.kernels import ops
from delta_b200.parts.base import FEED_FORWARDS, MIXERS, RunState, PartSpec

DEVICE = "cuda:0"
PAGE = 16
EPS = 1e-5
F64 = torch.float64


# ------------------------------------------------------------------ the cases

def listed():
    return [
        # The headline: a decode step of a Yi-6B-sized model (4 of its 32 layers) at batch 8 and context 4,096, replayed from its graph.
        dict(name="yi_decode", kind="yi_decode", width=4096, layers=4, batch=8, context=4096, vocab=64000),
        # The attention layer of a 2,048-token Yi-6B prompt (projections, rotary positions, paged cache, tcgen05 attention).
        dict(name="yi_attention_prompt", kind="yi_attention", width=4096, rows="2048", cached=0),
        # The SwiGLU feed-forward of the same prompt: the largest share of a dense model's prefill.
        dict(name="yi_mlp_prompt", kind="yi_mlp", width=4096, intermediate=11008, rows="2048"),
        # A mixture of 16 experts (4 chosen, clamped gates, a shared expert) over a 2,048-token prompt at width 2,048.
        dict(name="experts_prompt", kind="experts", width=2048, style="clamped", rows="2048", decode=False),
        # The same design's decode step at batch 8, from a graph: nearly every expert's weights are read for eight tokens.
        dict(name="experts_decode", kind="experts", width=2048, style="clamped", rows="1,1,1,1,1,1,1,1", decode=True),
        # Latent attention (16 heads, latent 256 + 64 rotated entries) over a 2,048-token prompt.
        dict(name="latent_prompt", kind="latent", width=2048, rows="2048", cached=0, window=0, decode=False),
        # The same layer's decode step at batch 8 and context 2,048, from a graph: the smallest call.
        dict(name="latent_decode", kind="latent", width=2048, rows="1,1,1,1,1,1,1,1", cached=2047, window=0, decode=True),
        # Attention with capped scores, biases by distance and sinks over three prompts of odd lengths in one step.
        dict(name="shaped_prompt", kind="shaped", width=2048, rows="1301,700,47", cached=0),
        # Linear attention with a decay per head over a 2,048-token prompt: 16 heads of 128 x 128.
        dict(name="decay_prompt", kind="decay", width=2048, rows="2048"),
        # The gated delta rule over two prompts of odd lengths.
        dict(name="delta_prompt", kind="delta", width=2048, rows="1301,747"),
        # The state-space recurrence over a 2,048-token prompt: 64 heads of 64 channels and 128 states.
        dict(name="state_space_prompt", kind="state_space", width=2048, rows="2048"),
        # The 32-bit path: a 300-token prompt through a small Yi model, logits of every token.
        dict(name="yi_prompt_f32", kind="yi_prompt_f32", width=2048, layers=2, rows="300", vocab=32000),
    ]


def _cut(rng, total, most):
    """``total`` tokens cut into up to ``most`` rows of odd lengths."""
    n = rng.randint(1, most)
    cuts = sorted(rng.sample(range(1, total), n - 1)) if n > 1 else []
    return ",".join(str(b - a) for a, b in zip([0] + cuts, cuts + [total]))


def _log(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(("yi_decode", "yi_attention", "yi_mlp", "experts", "experts", "latent", "latent", "shaped", "decay", "delta",
                       "state_space", "yi_prompt_f32"))
    tokens = _log(rng, 65, 2048)
    if kind == "yi_decode":
        return dict(kind=kind, width=rng.choice((2048, 4096)), layers=rng.randint(1, 4), batch=rng.randint(1, 16), context=_log(rng, 64, 4096),
                    vocab=rng.choice((32000, 64000)))
    if kind == "yi_attention":
        return dict(kind=kind, width=rng.choice((2048, 4096)), rows=_cut(rng, tokens, 4), cached=rng.choice((0, 0, rng.randint(1, 2048))))
    if kind == "yi_mlp":
        return dict(kind=kind, width=4096, intermediate=11008, rows=str(tokens))
    if kind == "experts":
        decode = rng.random() < 0.4
        rows = ",".join(["1"] * rng.randint(1, 32)) if decode else _cut(rng, tokens, 4)
        return dict(kind=kind, width=rng.choice((1024, 2048)), style=rng.choice(("clamped", "relu_squared")), rows=rows, decode=decode)
    if kind == "latent":
        decode = rng.random() < 0.4
        rows = ",".join(["1"] * rng.randint(1, 16)) if decode else _cut(rng, tokens, 4)
        return dict(kind=kind, width=rng.choice((1024, 2048)), rows=rows, cached=_log(rng, 16, 4000) if decode else rng.choice((0, 0, rng.randint(1, 2048))),
                    window=rng.choice((0, 0, 1024)), decode=decode)
    if kind == "shaped":
        return dict(kind=kind, width=rng.choice((1024, 2048)), rows=_cut(rng, tokens, 4), cached=rng.choice((0, 0, rng.randint(1, 1024))))
    if kind == "yi_prompt_f32":
        return dict(kind=kind, width=rng.choice((1024, 2048)), layers=rng.randint(1, 2), rows=_cut(rng, _log(rng, 17, 300), 2), vocab=32000)
    return dict(kind=kind, width=rng.choice((1024, 2048)), rows=_cut(rng, tokens, 4))


# ------------------------------------------------------------------ sizes

def _rows(case):
    return [int(n) for n in str(case.get("rows", "1")).split(",")]


def _part(case):
    """(registry, kind, parameters) of the layer: the sizes of the benchmark's models at this width."""
    d, k = case["width"], case["kind"]
    H = d // 128
    if k == "yi_attention":
        return MIXERS, "gqa_attention", dict(prefix="", width=d, heads=d // 128, kv_heads=max(1, d // 1024), head_dim=128, position=PartSpec(
            "rotary", dict(head_dim=128, theta=5e6, max_positions=8192), "position"))
    if k == "yi_mlp":
        return FEED_FORWARDS, "swiglu", dict(prefix="", width=d, intermediate=case["intermediate"])
    if k == "experts" and case["style"] == "clamped":
        return FEED_FORWARDS, "experts", dict(prefix="", width=d, experts=16, top=4, intermediate=d // 2, limit=7.0,
                                              shared=dict(intermediate=d // 2, limit=7.0))
    if k == "experts":
        return FEED_FORWARDS, "experts", dict(prefix="", width=d, experts=16, top=4, intermediate=d // 2, scoring="sigmoid", correction=True,
                                              route_scale=2.5, activation="relu_squared", wide_output=True)
    if k == "latent":
        return MIXERS, "latent_attention", dict(
            prefix="", width=d, heads=H, head_dim=128, rot_dim=64, value_dim=128, kv_rank=256, eps=EPS, scale=0.07, window=case["window"] or None,
            position=PartSpec("rotary", dict(head_dim=64, theta=500000.0, max_positions=8192, interleaved=False), "position"), rot_dims=64)
    if k == "shaped":
        return MIXERS, "sink_attention", dict(
            prefix="", width=d, heads=H, kv_heads=max(1, H // 4), head_dim=128, value_dim=128, scale=0.09, sink=True, bias=True, out_bias=False,
            qk_norm_eps=EPS, qk_norm_whole=True, q_temp=dict(coef=0.1, every=512), softcap=50.0, distance_bias=dict(rows=32, far=1024))
    if k == "decay":
        return MIXERS, "decay_attention", dict(prefix="", width=d, heads=H, head_dim=128, value_dim=128, decays=_decays(H), eps=EPS)
    if k == "delta":
        return MIXERS, "channel_delta", dict(prefix="", width=d, heads=H, kv_heads=H, head_dim=128, value_dim=128, conv=4, decay_rank=128,
                                             gate_rank=128, eps=EPS)
    if k == "state_space":
        return MIXERS, "state_space", dict(prefix="", width=d, heads=d // 32, head_dim=64, state=128, groups=2, conv=4, norm_groups=1, eps=EPS)
    raise ValueError(k)


def _decays(H):
    return [1.0 - 2.0 ** (-5 - 3 * h / max(1, H - 1)) for h in range(H)]


def _yi(case):
    d = case["width"]
    return dict(architectures=["YiForCausalLM"], hidden_size=d, num_hidden_layers=case["layers"], num_attention_heads=d // 128,
                num_key_value_heads=max(1, d // 1024), intermediate_size=11008 * d // 4096, vocab_size=case["vocab"], rms_norm_eps=1e-5,
                rope_theta=5e6, max_position_embeddings=8192, model_type="llama")


# ------------------------------------------------------------------ inputs, from the seed alone

def _gen(name, seed):
    g = torch.Generator(device=DEVICE)
    g.manual_seed((zlib.crc32(name.encode()) * 1000003 + int(seed)) % (1 << 62))
    return g


class Weights:
    """Tensors by name, the same for whoever asks with this seed: matrices N(0, 0.02) in the compute type, vectors in 32 bit."""

    def __init__(self, seed, dtype=torch.bfloat16):
        self.seed, self.dtype = seed, dtype

    def __call__(self, name, shape, init="normal"):
        g = _gen("w:" + name, self.seed)
        if init == "normal":
            return torch.randn(shape, generator=g, device=DEVICE).mul_(0.02).to(self.dtype)
        low, high = (0.9, 1.1) if init == "norm" else (float(v) for v in init.split(":")[1:3])
        return torch.rand(shape, generator=g, device=DEVICE) * (high - low) + low

    def of(self, specs):
        return {s.name: self(s.name, tuple(s.shape), s.init) for s in specs}


def _inputs(case, seed):
    """Rows as a norm hands them on."""
    return torch.randn((sum(_rows(case)), case["width"]), generator=_gen("x", seed), device=DEVICE).to(torch.bfloat16)


def _cached(name, seed, shape):
    """What earlier steps left in the cache: rotated keys, values and normed latents are all about N(0, 1)."""
    return torch.randn(shape, generator=_gen(name, seed), device=DEVICE).to(torch.bfloat16)


def _fill_pages(cache, cid, slots, held):
    """``held`` [rows, tokens of whole pages, ...]: a layer's cached tokens, the token axis second; written where the requests' pages lie."""
    g = cache.group_of_cache[cid]
    n = held.shape[1] // PAGE
    table = torch.as_tensor(g.table[slots, :n].astype(np.int64), device=DEVICE).reshape(-1)
    pages = cache.layer_pages(cid)
    rows = held.view(len(slots) * n, PAGE, *held.shape[2:])
    if rows.dim() == 5:      # [page, token, 2, kv head, entry] -> [page, 2, kv head, token, entry]
        rows = rows.permute(0, 2, 3, 1, 4)
    elif rows.dim() == 4:    # [page, token, kv head, entry] -> [page, kv head, token, entry]
        rows = rows.permute(0, 2, 1, 3)
    pages[table] = rows.to(pages.dtype)


def _whole_pages(n):
    return (n + PAGE - 1) // PAGE * PAGE


# ------------------------------------------------------------------ what a program has in hand

class Layer:
    """One part with its weights, its cache and the rows of a step."""

    def __init__(self, case, seed):
        registry, kind, params = _part(case)
        self.case, self.rows, self.done = case, _rows(case), int(case.get("cached", 0))
        self.part = registry.create(kind, **params)
        self.part.bind(Weights(seed).of(self.part.tensor_specs()))
        self.x = _inputs(case, seed)
        mixer = registry is MIXERS
        spec = self.part.cache_spec() if mixer else None
        states = self.part.run_state_specs() if hasattr(self.part, "run_state_specs") else {}
        most = self.done + max(self.rows)
        pages = len(self.rows) * (_whole_pages(most) // PAGE + 8)
        self.cache = CacheManager({0: spec} if spec else {}, states, max_slots=len(self.rows), max_seq_len=most, page_size=PAGE, num_pages=pages,
                                  dtype=torch.bfloat16, device=torch.device(DEVICE))
        self.slots = [self.cache.acquire_slot() for _ in self.rows]
        for s, n in zip(self.slots, self.rows):
            self.cache.grow(s, self.done + n)
        if self.done:      # whole pages behind the context too: the new tokens overwrite them
            n = self.done // PAGE * PAGE
            self.held = _held(case, seed)
            _fill_pages(self.cache, 0, self.slots, self.held[:, :n].contiguous())
            if self.done > n:
                tail = torch.zeros((len(self.rows), PAGE, *self.held.shape[2:]), dtype=torch.bfloat16, device=DEVICE)
                tail[:, :self.done - n] = self.held[:, n:]
                self._tail(n // PAGE, tail)
        self.err = ops.new_error_record(torch.device(DEVICE))
        self.scratch = {}
        self.has_cache, self.has_state = spec is not None, bool(states)
        self.sections, self.tables = self._device_rows()
        self.graph = None
        if case.get("decode"):
            self._record()

    def _tail(self, page, rows):
        """The page that the context ends in."""
        g = self.cache.group_of_cache[0]
        at = torch.as_tensor(g.table[self.slots, page].astype(np.int64), device=DEVICE)
        pages = self.cache.layer_pages(0)
        rows = rows.permute(0, 2, 3, 1, 4) if rows.dim() == 5 else rows.permute(0, 2, 1, 3)
        pages[at] = rows

    def _device_rows(self):
        i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEVICE)      # noqa: E731
        n = self.rows
        starts = [sum(n[:i]) for i in range(len(n))]
        s = dict(tokens=i32([0] * sum(n)), tok_row=i32([r for r, k in enumerate(n) for _ in range(k)]),
                 tok_pos=i32([self.done + p for k in n for p in range(k)]), row_slot=i32(self.slots), row_flags=i32([0] * len(n)),
                 row_q_start=i32(starts), row_q_len=i32(n), row_pos_start=i32([self.done] * len(n)), logit_rows=i32([]))
        self.starts = starts
        self.width = max(1, self.cache.max_pages_per_request)
        tables = {name: i32(g.table[self.slots, :self.width].tolist()) for name, g in self.cache.groups.items()}
        return s, tables

    def context(self, replayable=False):
        n = self.rows
        host = dict(max_pages=self.width, decode_only=all(k == 1 for k in n), max_q_len=max(n), max_seq_len=self.done + max(n),
                    rows=[RowInput(s, [0] * k, self.done) for s, k in zip(self.slots, n)], q_lens=list(n), q_start=list(self.starts), wants=[])
        return StepContext(device=torch.device(DEVICE), dtype=torch.bfloat16, cache=self.cache, sections=self.sections, block_tables=self.tables,
                           host=host, err=self.err, scratch_pool=self.scratch, replayable=replayable, max_rows=len(n), max_step_tokens=2048)

    def forward(self, ctx):
        if self.has_state:
            for t in self.cache.states.values():
                t.zero_()
            return (self.part.forward(ctx, self.x, RunState(self.cache.states)), dict(self.cache.states))
        if self.has_cache:
            return self.part.forward(ctx, self.x, ctx.cache_view(0, True)), self.cache.layer_pages(0)
        return self.part.forward(ctx, self.x)

    def _record(self):
        for _ in range(2):
            self.forward(self.context(replayable=True))
        torch.cuda.synchronize()
        self.graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(self.graph):
            self.out = self.forward(self.context(replayable=True))

    def run(self):
        if self.graph is not None:
            self.graph.replay()
            return self.out
        return self.forward(self.context())


def _held(case, seed):
    rows, done = len(_rows(case)), case["cached"]
    d, k = case["width"], case["kind"]
    shape = {"yi_attention": (2, max(1, d // 1024), 128), "latent": (1, 320), "shaped": (max(1, d // 512), 256)}[k]
    return _cached("held", seed, (rows, done) + shape)


class YiDecode:
    """A Yi engine whose requests have ``context - 1`` tokens cached, about to decode one more each."""

    def __init__(self, case, seed):
        B, n, L = case["batch"], case["context"], case["layers"]
        self.layers = L
        cfg = EngineConfig(max_batch=B, max_seq_len=_whole_pages(n), page_size=PAGE, num_pages=B * (_whole_pages(n) // PAGE + 8), cuda_graph_decode=True)
        self.runner = ModelRunner(config_json=_yi(case), seed=0, engine_config=cfg)
        self.runner.model.bind(Weights(seed).of(self.runner.model.tensor_specs()))
        self.slots = [self.runner.cache.acquire_slot() for _ in range(B)]
        for s in self.slots:
            self.runner.cache.grow(s, n)
        for layer in range(L):
            _fill_pages(self.runner.cache, layer, self.slots, _yi_held(case, seed, layer))
        self.rows = [RowInput(s, [t], n - 1, [0]) for s, t in zip(self.slots, _tokens(case, seed, B))]
        for _ in range(3):      # two eager runs, then the recording
            self.runner.step_and_sample(self.rows)
        torch.cuda.synchronize()

    def run(self):
        logits, tokens = self.runner.step_and_sample(self.rows)
        return logits, [self.runner.cache.layer_pages(i) for i in range(self.layers)]


def _yi_held(case, seed, layer):
    return _cached(f"held{layer}", seed, (case["batch"], _whole_pages(case["context"]), 2, max(1, case["width"] // 1024), 128))


def _tokens(case, seed, n):
    return torch.randint(0, case["vocab"], (n,), generator=_gen("tokens", seed), device=DEVICE).tolist()


class YiPromptF32:
    def __init__(self, case, seed):
        self.lens, self.layers = _rows(case), case["layers"]
        most = _whole_pages(max(self.lens))
        cfg = EngineConfig(max_batch=len(self.lens), max_seq_len=most, page_size=PAGE, dtype="float32")
        self.runner = ModelRunner(config_json=_yi(case), seed=0, engine_config=cfg)
        self.runner.model.bind(Weights(seed, torch.float32).of(self.runner.model.tensor_specs()))
        tokens = _tokens(case, seed, sum(self.lens))
        self.rows, at = [], 0
        for n in self.lens:
            slot = self.runner.cache.acquire_slot()
            self.runner.cache.grow(slot, n)
            self.rows.append(RowInput(slot, tokens[at:at + n], 0, list(range(n))))
            at += n

    def run(self):
        return self.runner.step(self.rows), [self.runner.cache.layer_pages(i) for i in range(self.layers)]


def prepare(case, seed):
    if case["kind"] == "yi_decode":
        return YiDecode(case, seed)
    if case["kind"] == "yi_prompt_f32":
        return YiPromptF32(case, seed)
    return Layer(case, seed)


def run(state):
    return state.run()


# ------------------------------------------------------------------ what a pass cannot do without

def work(case):
    d, k = case["width"], case["kind"]
    H = d // 128
    if k in ("yi_decode", "yi_prompt_f32"):
        G, inter, V, L = max(1, d // 1024), 11008 * d // 4096, case["vocab"], case["layers"]
        weights = L * (d * (H + 2 * G) * 128 + d * H * 128 + 3 * d * inter) + V * d
        if k == "yi_decode":
            T, es, pairs = case["batch"], 2, case["batch"] * case["context"]
            cache = pairs * L * 2 * G * 128
        else:
            T, es, pairs = sum(_rows(case)), 4, sum(n * (n + 1) // 2 for n in _rows(case))
            cache = T * L * 2 * G * 128
        return dict(bytes=es * (weights + cache + T * d) + 4 * T * V, flops=2 * T * weights + 4 * L * pairs * H * 128)
    n, done = _rows(case), int(case.get("cached", 0))
    T = sum(n)
    window = int(case.get("window", 0))
    reach = [(p, min(p + 1, window) if window else p + 1) for k_ in n for p in range(done, done + k_)]
    pairs = sum(r for _, r in reach)
    read = sum(min(done, window - 1) if window else done for _ in n)      # cached tokens that a row reads

    def result(weights, flops, extra=0):
        return dict(bytes=2 * weights + 4 * T * d + extra, flops=flops)
    if k == "yi_attention":
        G = max(1, d // 1024)
        w = d * (2 * H + 2 * G) * 128
        return result(w, 2 * T * w + 4 * pairs * H * 128, 4 * G * 128 * (read + T))
    if k == "yi_mlp":
        w = 3 * d * case["intermediate"]
        return result(w, 2 * T * w)
    if k == "experts":
        mats, shared = (3, 1) if case["style"] == "clamped" else (2, 0)
        each = mats * d * (d // 2)
        used = 16 * (1 - (1 - 4 / 16) ** T)      # experts that some token chooses, on average
        return result(used * each + shared * each, 2 * T * (4 + shared) * each)
    if k == "latent":
        w = d * (H * 192 + 320) + H * 128 * 256 * 2 + d * H * 128
        return result(w, 2 * T * w + 2 * pairs * H * (192 + 128), 2 * 320 * (read + T))
    if k == "shaped":
        G = max(1, H // 4)
        w = d * (H + 2 * G) * 128 + d * H * 128
        return result(w, 2 * T * w + 4 * pairs * H * 128, 2 * 256 * G * (read + T))
    if k == "decay":
        w = 5 * d * d
        return result(w, 2 * T * w + 4 * T * H * 128 * 128, 4 * len(n) * H * 128 * 128)
    if k == "delta":
        w = 4 * d * d + d * H + 2 * 128 * d * 2
        return result(w, 2 * T * w + 6 * T * H * 128 * 128, 4 * len(n) * H * 128 * 128)
    C, N, Hs = 2 * d, 128, d // 32
    w = d * (2 * C + 4 * N + Hs) + d * C
    return result(w, 2 * T * w + 4 * T * C * N, 4 * len(n) * C * N)


def tolerance(case):
    """Four times what the path shows against ``exact``, by kind."""
    return {"rel": {"yi_prompt_f32": 1.5e-5, "yi_decode": 6e-2, "yi_attention": 2e-2, "shaped": 2e-2, "delta": 1.8e-2}.get(case["kind"], 1.5e-2)}


# ------------------------------------------------------------------ the same in 64 bits

def _lin(x, w):
    return x @ w.to(F64).t()


def _rms(x, eps=EPS):
    return x / torch.sqrt((x * x).mean(-1, keepdim=True) + eps)


def _silu(x):
    return x * torch.sigmoid(x)


def _turn(x, pos, base, dims, half):
    """x [T, heads, n]: entries i and i + half of the first ``dims`` are turned by pos * base^(-2 i / dims)."""
    f = float(base) ** (-2.0 * torch.arange(half, dtype=F64, device=DEVICE) / dims)
    a = pos.to(F64)[:, None, None] * f
    c, s = torch.cos(a), torch.sin(a)
    u, v = x[..., :half], x[..., half:dims]
    return torch.cat([u * c - v * s, v * c + u * s, x[..., dims:]], dim=-1)


def _attend(q, k, v, start, scale, window=0, sink=None, shape=None):
    """q [T, H, dk] at positions start.., k [n, H, dk], v [n, H, dv], causal; a head at a time."""
    T, H = q.shape[:2]
    out = torch.empty((T, H, v.shape[-1]), dtype=F64, device=DEVICE)
    dist = (start + torch.arange(T, device=DEVICE))[:, None] - torch.arange(k.shape[0], device=DEVICE)[None, :]
    hidden = (dist < 0) | (dist >= window if window else dist < 0)
    for h in range(H):
        s = q[:, h] @ k[:, h].t() * scale
        s = (shape(s, h, dist) if shape is not None else s).masked_fill(hidden, -math.inf)
        if sink is not None:
            s = torch.cat([s, sink[h].to(F64).expand(T, 1)], dim=1)
        out[:, h] = torch.softmax(s, dim=-1)[:, :k.shape[0]] @ v[:, h]
    return out


def _by_row(case):
    at = 0
    for r, n in enumerate(_rows(case)):
        yield r, slice(at, at + n), n
        at += n


def _conv(x, w, b=None):
    taps = w.shape[1]
    p = torch.cat([torch.zeros((taps - 1, x.shape[1]), dtype=F64, device=DEVICE), x])
    y = sum(p[j:j + x.shape[0]] * w[:, j].to(F64) for j in range(taps))
    return y if b is None else y + b.to(F64)


def _exact_yi_layer(W, x, H, G, pos, p, held, inter, cut):
    """One pre-norm layer.  ``held``: per row keys and values [tokens, 2, G, 128] before it or None."""
    d = x.shape[1]
    h = _rms(x) * W(p + "input_layernorm.weight", (d,), "norm").to(F64)
    a = _exact_gqa(W, h, H, G, pos, p + "self_attn.", held, cut)
    x = x + a
    h = _rms(x) * W(p + "post_attention_layernorm.weight", (d,), "norm").to(F64)
    return x + _exact_swiglu(W, h, inter, p + "mlp.")


def _exact_gqa(W, h, H, G, pos, p, held, cut):
    d, T = h.shape[1], h.shape[0]
    q = _turn(_lin(h, W(p + "q_proj.weight", (H * 128, d))).view(T, H, 128), pos, 5e6, 128, 64)
    k = _turn(_lin(h, W(p + "k_proj.weight", (G * 128, d))).view(T, G, 128), pos, 5e6, 128, 64)
    v = _lin(h, W(p + "v_proj.weight", (G * 128, d))).view(T, G, 128)
    out = torch.empty((T, H, 128), dtype=F64, device=DEVICE)
    for r, (a, b) in enumerate(cut):
        kr, vr, done = k[a:b], v[a:b], 0
        if held is not None:
            done = held[r].shape[0]
            kr, vr = torch.cat([held[r][:, 0].to(F64), kr]), torch.cat([held[r][:, 1].to(F64), vr])
        out[a:b] = _attend(q[a:b], kr.repeat_interleave(H // G, 1), vr.repeat_interleave(H // G, 1), done, 128 ** -0.5)
    return _lin(out.reshape(T, H * 128), W(p + "o_proj.weight", (d, H * 128)))


def _exact_swiglu(W, h, inter, p):
    d = h.shape[1]
    a = _silu(_lin(h, W(p + "gate_proj.weight", (inter, d)))) * _lin(h, W(p + "up_proj.weight", (inter, d)))
    return _lin(a, W(p + "down_proj.weight", (d, inter)))


def _exact_yi(case, seed):
    d = case["width"]
    H, G, inter, V = d // 128, max(1, d // 1024), 11008 * d // 4096, case["vocab"]
    if case["kind"] == "yi_decode":
        B, n = case["batch"], case["context"]
        W, tokens, cut = Weights(seed), _tokens(case, seed, B), [(b, b + 1) for b in range(B)]
        pos = torch.full((B,), n - 1, device=DEVICE)
    else:
        lens = _rows(case)
        W, tokens = Weights(seed, torch.float32), _tokens(case, seed, sum(lens))
        cut = [(sum(lens[:i]), sum(lens[:i + 1])) for i in range(len(lens))]
        pos = torch.cat([torch.arange(k, device=DEVICE) for k in lens])
    x = W("model.embed_tokens.weight", (V, d)).to(F64)[torch.tensor(tokens, device=DEVICE)]
    for i in range(case["layers"]):
        held = [t[:n - 1] for t in _yi_held(case, seed, i)] if case["kind"] == "yi_decode" else None
        x = _exact_yi_layer(W, x, H, G, pos, f"model.layers.{i}.", held, inter, cut)
    h = _rms(x) * W("model.norm.weight", (d,), "norm").to(F64)
    return _lin(h, W("lm_head.weight", (V, d)))


def _exact_experts(case, W, x):
    d, F = case["width"], case["width"] // 2
    clamped = case["style"] == "clamped"
    z = _lin(x, W("router", (16, d)))
    if clamped:
        weight, chosen = torch.topk(z, 4, dim=-1)
        weight = torch.softmax(weight, dim=-1)
    else:
        s = torch.sigmoid(z)
        chosen = torch.topk(s + W("correction", (16,), "uniform:-0.2:0.2").to(F64), 4, dim=-1).indices
        weight = torch.gather(s, 1, chosen)
        weight = 2.5 * weight / (weight.sum(-1, keepdim=True) + 1e-20)

    def one(h, p):
        if not clamped:
            return _lin(torch.relu(_lin(h, W(p + "up", (F, d)))) ** 2, W(p + "down", (d, F)))
        g, u = _lin(h, W(p + "gate", (F, d))).clamp(max=7.0), _lin(h, W(p + "up", (F, d))).clamp(-7.0, 7.0)
        return _lin(g * torch.sigmoid(1.702 * g) * (u + 1.0), W(p + "down", (d, F)))
    out = torch.zeros_like(x)
    for e in range(16):
        t, j = (chosen == e).nonzero(as_tuple=True)
        if t.numel():
            out[t] += weight[t, j][:, None] * one(x[t], f"e{e}.")
    if clamped:
        out = out + torch.sigmoid(_lin(x, W("shared.sg", (1, d)))) * one(x, "shared.")
    return out


def _exact_latent(case, W, x, held):
    d, T = case["width"], x.shape[0]
    H, done = d // 128, case["cached"]
    q = _lin(x, W("q", (H * 192, d))).view(T, H, 192)
    low = _lin(x, W("dkv", (320, d)))
    c = _rms(low[:, :256]) * W("dkv.norm", (256,), "norm").to(F64)
    uk, uv = W("uk", (H * 128, 256)), W("uv", (H * 128, 256))
    out = torch.empty((T, H, 128), dtype=F64, device=DEVICE)
    for r, rows, n in _by_row(case):
        pos = done + torch.arange(n, device=DEVICE)
        qr = torch.cat([q[rows, :, :128], _turn(q[rows, :, 128:], pos, 500000.0, 64, 32)], dim=-1)
        lat, rot = c[rows], _turn(low[rows, None, 256:], pos, 500000.0, 64, 32)[:, 0]
        if done:
            lat, rot = torch.cat([held[r, :, 0, :256].to(F64), lat]), torch.cat([held[r, :, 0, 256:].to(F64), rot])
        k = torch.cat([_lin(lat, uk).view(-1, H, 128), rot[:, None].expand(-1, H, -1)], dim=-1)
        out[rows] = _attend(qr, k, _lin(lat, uv).view(-1, H, 128), done, 0.07, case["window"])
    return _lin(out.reshape(T, H * 128), W("o", (d, H * 128)))


def _exact_shaped(case, W, x, held):
    d, T = case["width"], x.shape[0]
    H, done = d // 128, case["cached"]
    G = max(1, H // 4)
    bias = "uniform:-0.1:0.1"
    q = _rms(_lin(x, W("q", (H * 128, d))) + W("q.b", (H * 128,), bias).to(F64)) * W("q.norm", (H * 128,), "norm").to(F64)
    k = _rms(_lin(x, W("k", (G * 128, d))) + W("k.b", (G * 128,), bias).to(F64)) * W("k.norm", (G * 128,), "norm").to(F64)
    v = _lin(x, W("v", (G * 128, d))) + W("v.b", (G * 128,), bias).to(F64)
    rel, sink = W("rel", (32, H), "uniform:-1:1").to(F64), W("sink", (H,), "uniform:-1:1")
    by = [n if n < 16 else min(31, 16 + int(math.floor(math.log(n / 16) / math.log(1024 / 16) * 16))) for n in range(1025)]
    by = torch.tensor(by, device=DEVICE)

    def shape(s, h, dist):
        return 50.0 * torch.tanh(s / 50.0) + rel[by[dist.clamp(0, 1024)], h]
    out = torch.empty((T, H, 128), dtype=F64, device=DEVICE)
    for r, rows, n in _by_row(case):
        pos = done + torch.arange(n, device=DEVICE)
        temp = 1.0 + 0.1 * torch.log(torch.floor((pos.to(F64) + 1.0) / 512.0) + 1.0)
        kr, vr = k[rows].view(n, G, 128), v[rows].view(n, G, 128)
        if done:
            kr, vr = torch.cat([held[r, :, :, :128].to(F64), kr]), torch.cat([held[r, :, :, 128:].to(F64), vr])
        out[rows] = _attend((q[rows] * temp[:, None]).view(n, H, 128), kr.repeat_interleave(H // G, 1), vr.repeat_interleave(H // G, 1), done, 0.09,
                            sink=sink, shape=shape)
    return _lin(out.reshape(T, H * 128), W("o", (d, H * 128)))


def _states(**named):
    """The rows' states with the spare slot's behind them, in the order in which slots are handed out (the first request gets slot 0)."""
    return {k: torch.cat([torch.stack(v), torch.zeros((1, *v[0].shape), dtype=F64, device=DEVICE)]) for k, v in named.items()}


def _exact_decay(case, W, x):
    d, T = case["width"], x.shape[0]
    H = d // 128
    q, k, v = (_silu(_lin(x, W(n, (d, d)))).view(T, H, 128) for n in "qkv")
    lam = torch.tensor(_decays(H), dtype=F64, device=DEVICE)[:, None, None]
    o, kept = torch.empty((T, H, 128), dtype=F64, device=DEVICE), []
    for r, rows, n in _by_row(case):
        S = torch.zeros((H, 128, 128), dtype=F64, device=DEVICE)
        for t in range(rows.start, rows.stop):
            S = lam * S + k[t][:, :, None] * v[t][:, None, :]
            o[t] = torch.einsum("hkv,hk->hv", S, q[t])
        kept.append(S)
    y = _rms(o.reshape(T, d)) * W("norm", (d,), "norm").to(F64) * torch.sigmoid(_lin(x, W("g", (d, d))))
    return _lin(y, W("o", (d, d))), _states(decay_attention=kept)


def _tails(case, raw, taps):
    """The convolution's last inputs of every row, oldest first; zeros before a row's start."""
    out = []
    for r, rows, n in _by_row(case):
        p = torch.cat([torch.zeros((taps - 1, raw.shape[1]), dtype=F64, device=DEVICE), raw[rows]])
        out.append(p[-(taps - 1):])
    return out


def _exact_delta(case, W, x):
    d, T = case["width"], x.shape[0]
    H = d // 128
    taps = "uniform:-0.5:0.5"
    raw = torch.cat([_lin(x, W(n, (d, d))) for n in "qkv"], dim=1)
    w = torch.cat([W(n + ".conv", (d, 4), taps) for n in "qkv"])
    unit = lambda t: t / torch.sqrt((t * t).sum(-1, keepdim=True) + 1e-6)      # noqa: E731
    beta = torch.sigmoid(_lin(x, W("b", (H, d))))
    a = _lin(_lin(x, W("a1", (128, d))), W("a2", (d, 128))) + W("dt_bias", (d,), "uniform:-5:-1").to(F64)
    g = torch.exp(-torch.exp(W("A_log", (H,), "uniform:0:2").to(F64))[None, :, None] * torch.nn.functional.softplus(a).view(T, H, 128))
    o, kept = torch.empty((T, H, 128), dtype=F64, device=DEVICE), []
    for r, rows, n in _by_row(case):
        q, k, v = (t.reshape(n, H, 128) for t in _silu(_conv(raw[rows], w)).split(d, dim=1))
        q, k = unit(q) / math.sqrt(128.0), unit(k)
        S = torch.zeros((H, 128, 128), dtype=F64, device=DEVICE)      # [head, key entry, value entry]
        for t in range(n):
            at = rows.start + t
            S = g[at][:, :, None] * S
            u = beta[at][:, None] * (v[t] - torch.einsum("hkv,hk->hv", S, k[t]))
            S = S + k[t][:, :, None] * u[:, None, :]
            o[at] = torch.einsum("hkv,hk->hv", S, q[t])
        kept.append(S.transpose(1, 2))
    gate = torch.sigmoid(_lin(_lin(x, W("g1", (128, d))), W("g2", (d, 128)))).view(T, H, 128)
    y = _rms(o) * W("norm", (128,), "norm").to(F64) * gate
    return _lin(y.reshape(T, d), W("o", (d, d))), _states(conv=_tails(case, raw, 4), delta=kept)


def _exact_state_space(case, W, x):
    d, T = case["width"], x.shape[0]
    H, P, N, G = d // 32, 64, 128, 2
    C = H * P
    ch = C + 2 * G * N
    z, raw, dt = torch.split(_lin(x, W("in", (C + ch + H, d))), [C, ch, H], dim=-1)
    w, b = W("conv", (ch, 4), "uniform:-0.5:0.5"), W("conv.b", (ch,), "uniform:-0.1:0.1")
    dt = torch.nn.functional.softplus(dt + W("dt_bias", (H,), "uniform:-5:-1").to(F64))
    A, D = torch.exp(W("A_log", (H,), "uniform:0:2").to(F64)), W("D", (H,), "norm").to(F64)
    y, kept = torch.empty((T, H, P), dtype=F64, device=DEVICE), []
    for r, rows, n in _by_row(case):
        u, B, Cm = torch.split(_silu(_conv(raw[rows], w, b)), [C, G * N, G * N], dim=-1)
        u = u.reshape(n, H, P)
        B, Cm = (t.reshape(n, G, N).repeat_interleave(H // G, dim=1) for t in (B, Cm))
        S = torch.zeros((H, P, N), dtype=F64, device=DEVICE)
        for t in range(n):
            at = rows.start + t
            S = torch.exp(-A * dt[at])[:, None, None] * S + u[t][:, :, None] * (dt[at][:, None] * B[t])[:, None, :]
            y[at] = torch.einsum("hpn,hn->hp", S, Cm[t]) + D[:, None] * u[t]
        kept.append(S)
    y = y.reshape(T, C) * _silu(z)
    return _lin(_rms(y) * W("norm", (C,), "norm").to(F64), W("o", (d, C))), _states(conv=_tails(case, raw, 4), ssd=kept)


@torch.no_grad()
def exact(case, seed):
    """What ``run`` returns, but for the cache's pages, which lie as the pool hands them out."""
    k = case["kind"]
    if k in ("yi_decode", "yi_prompt_f32"):
        return _exact_yi(case, seed), None
    W, x = Weights(seed), _inputs(case, seed).to(F64)
    held = _held(case, seed) if case.get("cached") else None
    if k == "yi_attention":
        d = case["width"]
        cut = [(s.start, s.stop) for _, s, _ in _by_row(case)]
        pos = torch.cat([case["cached"] + torch.arange(n, device=DEVICE) for n in _rows(case)])
        return _exact_gqa(W, x, d // 128, max(1, d // 1024), pos, "", held, cut), None
    if k == "yi_mlp":
        return _exact_swiglu(W, x, case["intermediate"], "")
    if k == "experts":
        return _exact_experts(case, W, x)
    if k == "latent":
        return _exact_latent(case, W, x, held), None
    if k == "shaped":
        return _exact_shaped(case, W, x, held), None
    return {"decay": _exact_decay, "delta": _exact_delta, "state_space": _exact_state_space}[k](case, W, x)
