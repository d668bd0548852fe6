"""The tcgen05 attention kernels over a cache of rows whose value is the front part of its key, at the edges of its tiles."""
import pytest

from test_gpu_row_attention import run_case

pytestmark = pytest.mark.gpu


@pytest.fixture
def wide_everywhere(monkeypatch):
    from delta_b200.kernels import ops
    from delta_b200.parts import row_attention
    monkeypatch.setattr(row_attention, "TC_MIN_TOKENS", 2)
    calls = []
    real = ops.attention_rows_wide

    def counted(*a):
        calls.append(1)
        return real(*a)
    monkeypatch.setattr(ops, "attention_rows_wide", counted)
    yield calls
    assert calls, "the kernel did not run"


@pytest.mark.parametrize("shape", [(4, 1, 320, 256), (3, 1, 264, 200), (2, 1, 136, 64), (4, 2, 192, 128)])
@pytest.mark.parametrize("ps", [8, 16, 64])
def test_wide_portions(wide_everywhere, shape, ps):
    """Tiles of 64 keys and 128 queries: one and many, rows of unequal lengths, contexts before them, windows and chunks that end inside tiles."""
    run_case("bfloat16", False, shape, [(0, 63), (33, 64), (0, 2), (100, 65), (15, 9)], latent=True, seed=1, ps=ps)
    run_case("bfloat16", False, shape, [(0, 300), (130, 129)], latent=True, use_sink=True, gated=True, seed=2, ps=ps)
    run_case("bfloat16", False, shape, [(500, 260), (3, 128)], latent=True, use_sink=True, window=200, seed=3, ps=ps)
    run_case("bfloat16", False, shape, [(500, 260), (3, 128)], latent=True, window=33, gated=True, seed=4, ps=ps)
    run_case("bfloat16", False, shape, [(0, 270), (290, 140), (129, 3)], latent=True, use_sink=True, chunk=100, seed=5, ps=ps)


def test_wide_many_pieces_beside_single_tokens(wide_everywhere):
    run_case("bfloat16", False, (16, 1, 320, 256), [(0, 900), (700, 1), (300, 700), (64, 128), (0, 1)], latent=True, use_sink=True, seed=6)


@pytest.mark.parametrize("kp", [0, 15, 63, 64, 127, 128, 255, 298])
def test_wide_one_key_that_matters(wide_everywhere, kp):
    run_case("bfloat16", False, (4, 1, 320, 256), [(150, 150)], latent=True, spikes=[(0, 149, kp)], seed=kp)
