"""32-bit products by tensor cores: tiles' and chunks' ends, the same bits whatever shares a step, numbers that the parts do not reach."""
import math

import pytest
import torch

from test_gpu_kernels import DEV, ops

pytestmark = pytest.mark.gpu


def run(a, w):
    o = ops()
    assert o.gemm_f32_tc_supported(w)
    out = torch.full((a.shape[0] + 1, w.shape[0]), 7.0, device=DEV)
    err = o.new_error_record(DEV)
    o.gemm_f32_tc(a, w, out[:-1], err=err)
    o.raise_if_error(err)
    assert bool((out[-1] == 7.0).all())
    return out[:-1]


# token tiles of 16 to 160, K beside a chunk of 64 and in segments of 4 to 10 chunks, fewer and more rows of W than a tile, more pieces than SMs,
# more rows than a launch takes
@pytest.mark.parametrize("M, N, K", [(1, 128, 1024), (16, 127, 1028), (17, 1, 1100), (33, 300, 2044), (49, 2049, 1080), (129, 4096, 4100), (161, 8200, 516),
                                     (300, 2560, 2048), (319, 11008, 512), (700, 9700, 1028), (16385, 40, 1024)])
def test_gemm_f32_tc(M, N, K):
    g = torch.Generator(device=DEV).manual_seed(M + N + K)
    a, w = torch.randn(M, K, device=DEV, generator=g), torch.randn(N, K, device=DEV, generator=g) * 0.05
    out = run(a, w)
    ref = a.double() @ w.double().T
    # parts and products left out: 2^-24 of a term; cut-off sums of a chunk and the rounded sum of K / 64 of them: (24 + K / 64) 2^-24 of the magnitudes bounds it by far
    bound = (26 + K // 64) * 2.0 ** -24 * (a.double().abs() @ w.double().abs().T)
    assert bool(((out.double() - ref).abs() <= bound).all())
    plain = torch.empty(M, N, device=DEV)
    ops().gemm_nt_plain(a, w, plain)
    assert (out.double() - ref).norm() <= (plain.double() - ref).norm()      # nearer than the chain of fused multiply-adds
    for m in (1, 2, 31, 100, 160, 299):
        if m < M:
            assert torch.equal(run(a[M - m:], w), out[M - m:]), m


@pytest.mark.parametrize("N", [300, 9500])      # K in segments, and as a whole
def test_gemm_f32_tc_numbers_out_of_the_parts_reach(N):
    """Infinite, NaN, very large and very small entries: the sums of the plain kernel for the rows that hold them, the others untouched."""
    g = torch.Generator(device=DEV).manual_seed(1)
    a, w = torch.randn(70, 1024, device=DEV, generator=g), torch.randn(N, 1024, device=DEV, generator=g)
    want = run(a, w)
    rows, cols = {3: math.inf, 9: -math.inf, 20: math.nan, 41: 3e38, 69: 1.5 * 2.0 ** 60}, {0: math.inf, 130: -3.3e38, 131: math.nan, 299: 2.0 ** 100}
    b, v = a.clone(), w.clone()
    for r, x in rows.items():
        b[r, (7 * r) % 1024] = x
    for r, x in cols.items():
        v[r, (5 * r) % 1024] = x
    b[50] *= 2.0 ** -60
    b[51] *= 2.0 ** -120
    b[52] = 0.0
    v[200] *= 2.0 ** -100
    v[201] = 0.0
    out, plain = run(b, v), torch.empty(70, N, device=DEV)
    ops().gemm_nt_plain(b, v, plain)
    odd_r, odd_c = list(rows) + [50, 51], list(cols) + [200]
    same = lambda x, y: torch.equal(torch.nan_to_num(x, nan=1.0), torch.nan_to_num(y, nan=1.0)) and torch.equal(x.isnan(), y.isnan())      # noqa: E731
    assert same(out[odd_r], plain[odd_r]) and same(out[:, odd_c], plain[:, odd_c])
    rest_r = [r for r in range(70) if r not in odd_r + [52]]
    rest_c = [c for c in range(N) if c not in odd_c + [201]]
    assert torch.equal(out[rest_r][:, rest_c], want[rest_r][:, rest_c])
    assert bool((out[52][rest_c] == 0).all()) and bool((out[rest_r][:, 201] == 0).all())


def test_gemm_f32_tc_refuses_what_it_does_not_take():
    o = ops()
    ok = torch.empty(8, 1024, device=DEV)
    assert o.gemm_f32_tc_supported(ok)
    for w in (torch.empty(8, 1020, device=DEV), torch.empty(8, 1026, device=DEV), torch.empty(8, 1024, device=DEV).bfloat16(), torch.empty(8193, device=DEV)[1:].view(8, 1024),
              torch.empty(1024, 8, device=DEV).T):
        assert not o.gemm_f32_tc_supported(w)
    with pytest.raises(o.KernelError):
        o.gemm_f32_tc(torch.empty(2, 1020, device=DEV), ok, torch.empty(2, 8, device=DEV))


@pytest.mark.parametrize("M, N, K", [(300, 2048, 2048), (300, 9600, 1024), (1, 12000, 2048), (161, 9500, 1028)])
def test_gemm_f32_tc_rows_out_of_reach_take_about_the_plain_kernels_time(M, N, K):
    """A prompt of rows that hold a NaN, and one whose weights do: the plain kernel's bits, without every output being summed by a thread of its own."""
    g = torch.Generator(device=DEV).manual_seed(4)
    a, w = torch.randn(M, K, device=DEV, generator=g), torch.randn(N, K, device=DEV, generator=g)
    a[:, 5] = math.nan
    a[M // 2, 5] = 2.0 ** 80
    w[N - 1, 3] = math.inf
    out, plain = torch.empty(M, N, device=DEV), torch.empty(M, N, device=DEV)
    o = ops()

    def took(f):
        f()
        best = math.inf
        for _ in range(5):
            e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            e0.record()
            f()
            e1.record()
            torch.cuda.synchronize()
            best = min(best, e0.elapsed_time(e1))
        return best
    t, p = took(lambda: o.gemm_f32_tc(a, w, out)), took(lambda: o.gemm_nt_plain(a, w, plain))
    assert torch.equal(torch.nan_to_num(out, nan=1.0), torch.nan_to_num(plain, nan=1.0)) and torch.equal(out.isnan(), plain.isnan())
    assert bool(out[M // 2, :N - 1].isfinite().all())
    print(f"{M} x {N} x {K}: {t * 1e3:.0f} us, plain {p * 1e3:.0f}")
    assert t < 4 * p + 0.2      # (a thread an output reads a row of W of its own, 4 bytes at a time: tens of times the plain kernel's time)


def one(bits):
    return torch.tensor([bits], dtype=torch.int32).view(torch.float32).item()


@pytest.mark.parametrize("N", [300, 9500])
def test_gemm_f32_tc_a_single_product_is_rounded_once(N):
    """Rows of one entry: the products left out are below 2^-24 of it, and the sum of those that are made is rounded once."""
    g = torch.Generator(device=DEV).manual_seed(2)
    K, M = 1024, 40
    at = torch.randint(0, K, (M,), device=DEV, generator=g)
    a = torch.zeros(M, K, device=DEV)
    a[torch.arange(M), at] = torch.randn(M, device=DEV, generator=g)
    w = torch.randn(N, K, device=DEV, generator=g)
    a[7, at[7]] = w[0] = one(0x3f80ffff)      # parts that are cut off leave 2^-7 and 2^-15 behind the first two
    out = run(a, w)
    ref = a.double() @ w.double().T
    assert bool(((out.double() - ref).abs() <= 2.0 ** -23 * ref.abs()).all())


@pytest.mark.parametrize("kind", ["one large entry", "four large entries", "few entries", "positive", "one sign a row"])
@pytest.mark.parametrize("N, K", [(600, 2048), (9600, 1024), (4100, 11008)])
def test_gemm_f32_tc_is_no_further_off_than_multiply_adds(kind, N, K):
    """Rows that a few entries dominate, and operands of one sign, where errors of one sign would add up: 2-norm and mean of the error against 64 bits."""
    g = torch.Generator(device=DEV).manual_seed(K)
    M = 64
    a, w = torch.randn(M, K, device=DEV, generator=g), torch.randn(N, K, device=DEV, generator=g) * 0.05
    far = torch.rand(M, K, device=DEV, generator=g)
    if kind == "one large entry":
        a.scatter_(1, far.topk(1).indices, 3000.0)
    elif kind == "four large entries":
        a.mul_(torch.where(far >= far.topk(4).values[:, -1:], 1000.0, 1.0))
    elif kind == "few entries":
        a.mul_(far >= far.topk(4).values[:, -1:])
    elif kind == "positive":
        a, w = far + 1.0, torch.rand(N, K, device=DEV, generator=g) + 1.0
    else:
        a, w = a.abs() * torch.where(torch.arange(M, device=DEV) % 2 == 0, 1.0, -1.0)[:, None], w.abs()
    out, plain = run(a, w), torch.empty(M, N, device=DEV)
    ops().gemm_nt_plain(a, w, plain)
    ref = a.double() @ w.double().T
    e, p = (out.double() - ref) / ref.norm(), (plain.double() - ref) / ref.norm()
    mean = ((out.double() - ref) / ref).mean()
    print(f"{kind} {N} x {K}: {e.norm():.3g} against {p.norm():.3g}, mean {mean:.3g}")
    # What is left out of a term is up to 2^-24 of it, 2^-26.5 in the mean square, beside its rounding of 2^-24.3: 2.3 % of the error where a row is hardly more
    # than a term.  Four terms are four roundings either way, here of a term's high parts' sum and there of a sum's: a quarter for that.
    assert e.norm() <= (1.25 if kind == "few entries" else 1.03) * p.norm()
    if kind in ("positive", "one sign a row"):
        # the relative error's mean: a chunk's sum is cut off after each of its four steps, at a quarter, half, three quarters and all of it, by half of 2^-23 on average
        # where its terms have more bits than the sum has room for
        assert mean.abs() <= 2.5 * 2.0 ** -24


@pytest.mark.parametrize("N", [300, 9500])
def test_gemm_f32_tc_small_entries_keep_their_bits(N):
    """Entries far below their row's largest, which the weights do not read: down to 2^-126 they have all of their 24 bits."""
    g = torch.Generator(device=DEV).manual_seed(3)
    K, M = 1024, 33
    a, w = torch.randn(M, K, device=DEV, generator=g), torch.zeros(N, K, device=DEV)
    col = torch.randint(0, K, (N,), device=DEV, generator=g)
    w[torch.arange(N), col] = 1.0 + torch.rand(N, device=DEV, generator=g)
    small = torch.rand(M, K, device=DEV, generator=g) < 0.5
    a[small] *= 2.0 ** -118
    out = run(a, w)
    ref = a.double() @ w.double().T
    held = ref.abs() >= 2.0 ** -124      # (a result below has fewer than 24 bits itself)
    assert bool(((out.double() - ref).abs() <= 2.0 ** -23 * ref.abs())[held].all()) and held.sum() > held.numel() // 2


def test_gemm_f32_tc_takes_its_memory_from_the_steps_pool():
    """One buffer for all products of a model's steps, made at the first step for the longest one."""
    from delta_b200.config import EngineConfig
    from delta_b200.engine.step import ModelRunner, RowInput
    config = dict(architectures=["YiForCausalLM"], model_type="llama", hidden_size=1024, num_hidden_layers=1, num_attention_heads=8, num_key_value_heads=2,
                  intermediate_size=2816, vocab_size=8000, rms_norm_eps=1e-5, rope_theta=5e6, max_position_embeddings=512)
    r = ModelRunner(config_json=config, seed=0, engine_config=EngineConfig(max_batch=2, max_seq_len=256, page_size=16, dtype="float32"))
    slot = r.cache.acquire_slot()
    r.cache.grow(slot, 256)
    r.step([RowInput(slot, list(range(5)), 0, [4])])
    buf = r._scratch["linear.f32"]
    assert buf.numel() >= ops().gemm_f32_tc_bytes(5, 8000, 1024)
    r.step([RowInput(slot, list(range(200)), 5, [199])])
    r.step([RowInput(slot, list(range(20)), 205, [0])])
    assert r._scratch["linear.f32"].data_ptr() == buf.data_ptr()
    with pytest.raises(ops().KernelError, match="working memory"):
        ops().gemm_f32_tc(torch.empty(2, 1024, device=DEV), torch.empty(8, 1024, device=DEV), torch.empty(2, 8, device=DEV),
                          work=torch.empty(1024, dtype=torch.uint8, device=DEV))
