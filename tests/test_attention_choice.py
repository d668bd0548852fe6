"""Which kernel takes a step's portions, where two of them could."""
import pytest


@pytest.mark.parametrize("q_lens, starts, heads, tiles", [
    ([2], [4000], 16, False), ([8], [4000], 16, False), ([16], [4000], 16, False), ([31], [4000], 16, True), ([31], [4000], 8, False),
    ([8] * 4, [1000] * 4, 16, True), ([2], [0], 16, False), ([128], [0], 16, True), ([300], [0], 16, True), ([300, 1, 1], [0, 4000, 4000], 16, True),
    ([2, 300], [4000, 0], 16, False), ([1, 1], [500, 500], 16, False), ([600], [4000], 32, True)])
def test_few_tokens_behind_a_long_context_stay_with_the_plain_kernel(q_lens, starts, heads, tiles):
    """A block of tiles walks all keys of its 32 queries alone: it pays once there are more single-token blocks than the device runs at once."""
    from delta_b200.parts.attention_kernels import tiles_pay
    assert tiles_pay(q_lens, starts, heads, 148) is tiles


@pytest.mark.parametrize("q_lens, heads, tiles", [([65], 8, False), ([65], 16, False), ([129], 16, False), ([257], 8, False), ([257], 16, True), ([500], 8, False),
                                                  ([500], 16, True), ([65] * 8, 8, True), ([2048], 2, False), ([2048], 16, True)])
def test_linear_attention_takes_long_chunks_where_they_fill_the_device(q_lens, heads, tiles):
    from delta_b200.parts.decay_attention import tiles_pay
    assert tiles_pay(q_lens, 64, heads, 148) is tiles


@pytest.mark.parametrize("q_lens, heads, tc", [
    ([65], 8, True), ([300] + [20] * 4, 16, True), ([65] + [1] * 16, 8, True), ([300], 32, True), ([1000], 16, True), ([2048], 16, True), ([65] * 8, 16, True), ([65] * 16, 8, True), ([500] * 4, 16, True),
    ([100] * 20, 16, True), ([130] * 15, 32, True), ([65] + [1] * 16, 16, False), ([65] + [1] * 32, 32, False), ([512] + [1] * 8, 16, False),
    ([512] + [1] * 32, 8, False), ([2000] + [1] * 32, 16, False), ([300] + [20] * 16, 16, False), ([2000, 20], 16, True)])
def test_linear_attention_leaves_the_tensor_cores_where_their_chunks_would_be_empty(q_lens, heads, tc):
    """A portion beside single tokens, each of which would be a chunk of 128 that holds an SM, and more of them than SMs."""
    from delta_b200.parts.decay_attention import tensor_cores_pay
    assert tensor_cores_pay(q_lens, 128, heads, 148) is tc


def test_linear_attentions_forms_share_their_working_memory(monkeypatch):
    """Steps of full chunks, of chunks that would be nearly empty and of few tokens, in any order: one buffer, as large as any of them asks for at the engine's limits."""
    from types import SimpleNamespace
    import torch
    from delta_b200.engine.context import StepContext
    from delta_b200.parts import decay_attention as part
    H, taken, steps = 16, [], [[2000] + [1] * 32, [2048], [65], [300, 300]]
    for name in ("decay_attention_tc", "decay_attention_tiles", "decay_attention_chunked"):
        monkeypatch.setattr(part.ops, name, lambda *a, name=name, **kw: taken.append(name))
    monkeypatch.setattr(part.ops, "gated_rms_norm", lambda *a, **kw: None)
    monkeypatch.setattr(part.linear, "linear", lambda ctx, x, w: torch.empty((x.shape[0], w), dtype=torch.bfloat16))
    for d, order in ((128, steps), (128, steps[::-1]), (64, steps), (64, steps[::-1])):
        mixer, pool = part.DecayAttention("", 2048, H, d, d, [0.9] * H, 1e-5), {}
        mixer.w_in, mixer.w_o = 4 * H * d, 2048
        for q_lens in order:
            ctx = SimpleNamespace(_scratch_pool=pool, device="cpu", host=dict(q_lens=q_lens), max_step_tokens=2048, max_rows=33, sm_count=148, replayable=False, decode_only=False,
                                  max_q_len=max(q_lens), err=None, row_slot=None, row_q_start=None, row_q_len=None, memo=lambda key, make: make())
            ctx.scratch = lambda *a, ctx=ctx, **kw: StepContext.scratch(ctx, *a, **kw)
            mixer.forward(ctx, torch.empty((sum(q_lens), 2048), dtype=torch.bfloat16), SimpleNamespace(state={part.STATE: None}))
        assert len(pool) == 1 and "__retired__" not in pool
        assert len(set(taken[-4:])) == 2
    assert set(taken) == {"decay_attention_tc", "decay_attention_tiles", "decay_attention_chunked"}
