"""The tcgen05 attention kernels over a cache of rows whose value is the front part of its key, and with shaped scores, at the edges of their tiles."""
import pytest
import torch

from test_gpu_row_attention import run_case

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


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


@pytest.mark.parametrize("dk, dv", [(128, 128), (64, 128), (72, 104)])
@pytest.mark.parametrize("cap, far", [(4.0, 37), (50.0, 400), (0.0, 64), (6.0, -1)])
def test_shaped_portions(dk, dv, cap, far):
    """Capped scores and biases by distance in the tcgen05 kernel (tiles beside, across and behind the table's last distance), beside the plain
    kernel's answer for the same inputs in 32 bit."""
    from delta_b200.kernels import ops
    g = torch.Generator().manual_seed(dk + far)
    H, KV, ps = 4, 2, 16
    lens, before = [130, 64, 300], [0, 200, 500]
    pages = [-(-(b + n) // ps) for b, n in zip(before, lens)]
    bt = torch.full((3, max(pages)), -1, dtype=torch.int32)
    order = torch.randperm(sum(pages), generator=g).to(torch.int32)
    for r in range(3):
        bt[r, :pages[r]] = order[sum(pages[:r]):sum(pages[:r + 1])]
    cache = torch.randn(sum(pages), KV, ps, dk + dv, generator=g).bfloat16()
    T = sum(lens)
    q = (torch.randn(T, H * dk, generator=g) * 1.5).bfloat16()
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)      # noqa: E731
    sink = torch.randn(H, generator=g).to(DEV)
    dist = (torch.randn(H, far + 1, generator=g) * 2).to(DEV) if far >= 0 else None
    rows = dict(block_table=bt.to(DEV), tok_row=i32([r for r, n in enumerate(lens) for _ in range(n)]),
                tok_pos=i32([b + j for b, n in zip(before, lens) for j in range(n)]), row_q_start=i32([sum(lens[:r]) for r in range(3)]),
                row_q_len=i32(lens), row_pos_start=i32(before), sink=sink, dist_bias=dist)
    got = {}
    for dtype in (torch.bfloat16, torch.float32):
        qd, cd = q.to(DEV).to(dtype), cache.to(DEV).to(dtype)
        out = torch.full((T, H * dv), float("nan"), dtype=dtype, device=DEV)
        err = ops.new_error_record(DEV)
        params = ops.row_attn_params(q=qd, cache=cd, q_stride=H * dk, q_head_stride=dk, out=out, H=H, KV=KV, dk=dk, dv=dv, ps=ps, row_width=dk + dv,
                                     k_off=0, v_off=dk, scale=0.1, softcap=cap, err=err, **rows)
        if dtype == torch.float32:
            ops.attention_rows_plain(params)
        else:
            assert ops.attention_rows_tc_supported(params)
            ops.attention_rows_tc(params, max(lens))
        ops.raise_if_error(err)
        got[dtype] = out.double()
    want = got[torch.float32]
    # weights to 16 bits, one rounding of the output to bfloat16 (2^-9 of it); values are about one
    assert (got[torch.bfloat16] - want).abs().max() < 2.0 ** -8 * want.abs().max()


# the persistent product's epilogue: columns that end beside a warp's 16 and its half of the tile, rows beside a tile's 128, every kind of result
@pytest.mark.parametrize("M, N", [(129, 8), (129, 136), (257, 264), (200, 392), (385, 520), (1300, 2056)])
@pytest.mark.parametrize("out_dtype", [torch.float32, torch.bfloat16])
def test_rows_product_writes_its_columns_and_no_others(M, N, out_dtype):
    from delta_b200.kernels import ops as o
    g = torch.Generator(device="cuda:0").manual_seed(M + N)
    x, w = torch.randn(M, 192, device="cuda:0", generator=g).bfloat16(), torch.randn(N, 192, device="cuda:0", generator=g).bfloat16()
    room = torch.full((M + 2, N), 5.0, dtype=out_dtype, device="cuda:0")
    err = o.new_error_record("cuda:0")
    o.gemm_tc(x, w, room[1:M + 1], err=err)
    o.raise_if_error(err)
    ref = x.double() @ w.double().T
    # 192 exact products summed in 32 bit; a bfloat16 result is rounded once more
    bound = 192 * 2.0 ** -23 * (x.double().abs() @ w.double().abs().T) + (2.0 ** -8 * ref.abs() if out_dtype == torch.bfloat16 else 0)
    assert bool(((room[1:M + 1].double() - ref).abs() <= bound).all()) and bool((room[0] == 5).all()) and bool((room[M + 1] == 5).all())


@pytest.mark.parametrize("H, dq, dr, R, rot, interleaved", [(16, 128, 64, 256, 64, False), (1, 8, 16, 8, 16, False), (5, 16, 24, 264, 16, True), (3, 64, 32, 512, 16, False),
                                                            (2, 8, 8, 520, 8, True), (4, 24, 16, 72, 8, False)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("apart", [False, True])
def test_latent_prepare_of_eight_entries_at_a_time(H, dq, dr, R, rot, interleaved, dtype, apart):
    """Latents below, at and above a warp's 256 and 512 entries (above: the general kernel), rotated parts that end inside the part, halves that are no whole
    number of eight (the general kernel), latents in rows of their own; tokens in pages out of order."""
    from delta_b200.kernels import ops as o
    g = torch.Generator().manual_seed(R + dr)
    T, ps, width = 19, 4, R + dr
    rows = torch.randn(T, H * (dq + dr) + (0 if apart else width), generator=g).to(dtype).to(DEV)
    low = torch.randn(T, width + 8, generator=g).to(dtype).to(DEV) if apart else None
    pos = torch.arange(T, dtype=torch.int32, device=DEV)
    bt = torch.randperm(5, generator=g).to(torch.int32).view(1, 5).to(DEV)
    angle = torch.arange(32, dtype=torch.float64)[:, None] * 100.0 ** (-2.0 * torch.arange(rot // 2, dtype=torch.float64) / rot)
    table = torch.stack([angle.cos(), angle.sin()], dim=-1).float().contiguous().to(DEV)
    w = (torch.rand(R, generator=g) + 0.5).to(DEV)
    cache = torch.full((6, 1, ps, width), 5.0, dtype=dtype, device=DEV)
    qabs = torch.full((T, H, width), 7.0, dtype=dtype, device=DEV)
    err = o.new_error_record(DEV)
    kw = dict(low=low, low_offset=8) if apart else {}
    o.latent_prepare(rows, pos, torch.zeros(T, dtype=torch.int32, device=DEV), bt, cache, qabs, norm_weight=w, eps=1e-5, H=H, dq=dq, dr=dr, R=R, ps=ps, table=table,
                     rot_dims=rot, interleaved=interleaved, err=err, **kw)
    o.raise_if_error(err)
    lat = (low[:, 8:] if apart else rows[:, H * (dq + dr):]).double()

    def turned(x):
        x = x.clone()
        c, s = table[:T, :, 0].double()[:, None], table[:T, :, 1].double()[:, None]
        a, b = (slice(0, rot, 2), slice(1, rot, 2)) if interleaved else (slice(0, rot // 2), slice(rot // 2, rot))
        u, v = x[..., a].clone(), x[..., b].clone()
        x[..., a], x[..., b] = u * c - v * s, v * c + u * s
        return x
    q = turned(rows[:, :H * (dq + dr)].double().view(T, H, dq + dr)[..., dq:])
    k = turned(lat[:, None, R:])[:, 0]
    c = lat[:, :R] / torch.sqrt((lat[:, :R] ** 2).mean(-1, keepdim=True) + 1e-5) * w.double()
    got = torch.stack([cache[bt[0, t // ps].item(), 0, t % ps] for t in range(T)]).double()
    tol = dict(atol=1e-2, rtol=2.0 ** -8) if dtype == torch.bfloat16 else dict(atol=2e-6, rtol=2e-6)      # one rounding of the result, a few of 32 bit
    assert torch.allclose(got, torch.cat([c, k], dim=1), **tol) and torch.allclose(qabs[..., R:].double(), q, **tol)
    assert bool((qabs[..., :R] == 7).all()) and bool((cache[5] == 5).all())


@pytest.mark.parametrize("H, dq, dr, R, rot, interleaved", [(16, 128, 64, 256, 64, False), (2, 8, 16, 8, 16, False), (3, 16, 24, 264, 16, True), (2, 64, 32, 512, 16, False)])
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
def test_latent_prepare_has_the_same_bits_from_either_kernel(H, dq, dr, R, rot, interleaved, dtype):
    """Latents that begin on a boundary of eight entries (eight at a time) and beside it (one at a time): norms and rotated parts are the same numbers."""
    from delta_b200.kernels import ops as o
    g = torch.Generator().manual_seed(R)
    T, ps, width = 300, 16, R + dr
    rows, lat = torch.randn(T, H * (dq + dr), generator=g).to(dtype).to(DEV), torch.randn(T, width, generator=g).to(dtype).to(DEV)
    angle = torch.arange(T, dtype=torch.float64)[:, None] * 100.0 ** (-2.0 * torch.arange(rot // 2, dtype=torch.float64) / rot)
    table = torch.stack([angle.cos(), angle.sin()], dim=-1).float().contiguous().to(DEV)
    w, bt = (torch.rand(R, generator=g) + 0.5).to(DEV), torch.arange(19, dtype=torch.int32, device=DEV).view(1, 19)
    got = []
    for off in (8, 3):
        low = torch.zeros(T, width + 8, dtype=dtype, device=DEV)
        low[:, off:off + width] = lat
        cache, qabs = torch.zeros((19, 1, ps, width), dtype=dtype, device=DEV), torch.zeros((T, H, width), dtype=dtype, device=DEV)
        o.latent_prepare(rows, torch.arange(T, dtype=torch.int32, device=DEV), torch.zeros(T, dtype=torch.int32, device=DEV), bt, cache, qabs, norm_weight=w, eps=1e-5,
                         H=H, dq=dq, dr=dr, R=R, ps=ps, table=table, rot_dims=rot, interleaved=interleaved, low=low, low_offset=off)
        got.append((cache, qabs))
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])
