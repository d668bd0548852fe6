"""Which kernel takes the rows of several tokens of a 32-bit step."""
import pytest


@pytest.mark.parametrize("q_lens, starts, heads, tiles", [
    ([2], [4000], 16, False), ([8], [4000], 16, False), ([16], [4000], 16, False), ([31], [4000], 16, True), ([31], [4000], 8, False),
    ([8] * 4, [1000] * 4, 16, True), ([2], [0], 16, False), ([128], [0], 16, True), ([300], [0], 16, True), ([300, 1, 1], [0, 4000, 4000], 16, True),
    ([2, 300], [4000, 0], 16, False), ([1, 1], [500, 500], 16, False), ([600], [4000], 32, True)])
def test_few_tokens_behind_a_long_context_stay_with_the_plain_kernel(q_lens, starts, heads, tiles):
    """A block of tiles walks all keys of its 32 queries alone: it pays once there are more single-token blocks than the device runs at once."""
    from delta_b200.parts.attention_kernels import tiles_pay
    assert tiles_pay(q_lens, starts, heads, 148) is tiles
