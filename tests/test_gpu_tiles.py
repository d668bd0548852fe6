"""Kernels at the sizes where their tiles can go wrong: one row or key beside a tile's edge, sizes below a tile, rows of very different lengths."""
import math

import pytest
import torch

from test_gpu_kernels import DEV, PagedCase, ops

pytestmark = pytest.mark.gpu


# 64 x 128, 32 x 64 and 32 x 32 sums a block, each with rows, columns and K beside the tiles' edges; the last two have no 16-byte rows
@pytest.mark.parametrize("M, N, K", [(300, 11012, 36), (1025, 2049, 20), (130, 11008, 132), (33, 2048, 64), (1, 65, 16), (65, 130, 18), (7, 33, 3)])
def test_gemm_f32_tiles(M, N, K):
    o = ops()
    torch.manual_seed(M + N)
    a, w = torch.randn(M, K, device=DEV), torch.randn(N, K, device=DEV)
    out = torch.full((M + 1, N), 7.0, device=DEV)
    o.gemm_nt_plain(a, w, out[:M])
    ref = a.double() @ w.double().T
    # a sum of K products, each rounded once: K / 2 units of 2^-24 of the sum of magnitudes bounds it by far
    bound = K * 2.0 ** -24 * (a.double().abs() @ w.double().abs().T) + 1e-30
    assert bool(((out[:M].double() - ref).abs() <= bound).all()) and bool((out[M:] == 7.0).all())
    one = torch.empty(1, N, device=DEV)
    o.gemm_nt_plain(a[M - 1:].contiguous(), w, one)      # another tile size, the same order of the sum
    assert torch.equal(one[0], out[M - 1])


@pytest.mark.parametrize("H, KV, hd, ps", [(4, 2, 128, 16), (3, 3, 64, 8), (8, 1, 32, 64)])
@pytest.mark.parametrize("window", [0, 1, 33, 100])
def test_attention_f32_tiles(H, KV, hd, ps, window):
    o = ops()
    case = PagedCase(torch.float32, H, KV, hd, ps, seq_lens=[2, 31, 32, 33, 200, 129, 97, 300], q_lens=[2, 31, 32, 33, 64, 2, 65, 1], seed=H + window)
    out, lse = torch.full((case.T, H * hd), 9.0, device=DEV), torch.empty(case.T, H, device=DEV)
    o.attention_f32(case.params(out, lse=lse, window=window), max(case.q_lens))
    ref, ref_lse, _ = case.reference(window=window)
    # scores of about 6 at most in 32 bit: their rounding (hd 2^-24 |q| |k| scale) moves a weight by less than 1e-5
    assert torch.allclose(out.cpu(), ref, atol=2e-5, rtol=2e-5)
    assert torch.allclose(lse.cpu(), ref_lse, atol=2e-5, rtol=2e-5)
    # the rows of one token are left to the plain kernel, the others give the same bits
    again = torch.full_like(out, 9.0)
    o.attention_f32(case.params(again, window=window, row_filter=2), max(case.q_lens))
    assert torch.equal(again[:-1], out[:-1]) and bool((again[-1] == 9.0).all())
    o.attention_plain(case.params(again, window=window, row_filter=1))
    assert torch.allclose(again[-1], out[-1], atol=2e-5, rtol=2e-5) and torch.equal(again[:-1], out[:-1])


def test_attention_f32_keeps_what_a_query_does_not_see_out_of_its_sums():
    """A later token's infinite value reaches its own query and the ones behind it only; a page outside the pool is reported and left out."""
    o = ops()
    case = PagedCase(torch.float32, 2, 1, 64, 16, seq_lens=[40], q_lens=[40], seed=5)
    page = int(case.bt[0, 1])
    case.kv[page, 1, 0, 4, 3] = math.inf      # position 20
    out = torch.empty(40, 128, device=DEV)
    o.attention_f32(case.params(out), 40)
    ref, _, _ = case.reference()
    assert torch.allclose(out[:20].cpu(), ref[:20], atol=2e-5, rtol=2e-5) and not bool(torch.isfinite(out[20:, 3]).any())
    case.bt[0, 1] = 1 << 20
    err = o.new_error_record(DEV)
    o.attention_f32(case.params(out, err=err), 40)
    with pytest.raises(o.KernelError, match="page id"):
        o.raise_if_error(err)
    assert torch.allclose(out[:16].cpu(), ref[:16], atol=2e-5, rtol=2e-5)


@pytest.mark.parametrize("M", [1, 7, 8, 9, 16])
@pytest.mark.parametrize("N, K, heads", [(256, 128, 16), (128, 256, 3), (40, 32, 5), (16, 160, 1)])
def test_gemm_heads(M, N, K, heads):
    """Operands of a head between those of the others, as they lie in a layer's rows; columns beside a warp's 16, K beside a step of 128."""
    o = ops()
    torch.manual_seed(M + N)
    a = torch.randn(M, heads, K + 8, device=DEV).bfloat16()
    w = (torch.randn(heads, N, K, device=DEV) * 0.1).bfloat16()
    c = torch.full((M, heads, N + 3), 5.0, dtype=torch.bfloat16, device=DEV)
    o.gemm_heads(a.data_ptr(), w.data_ptr(), c.data_ptr(), M, N, K, heads * (K + 8), heads * (N + 3), heads, K + 8, N * K, N + 3)
    ref = torch.einsum("mhk,hnk->mhn", a[:, :, :K].double(), w.double())
    # one rounding to bfloat16 (2^-9 of the value) and the rounding of a 32-bit sum
    assert bool(((c[:, :, :N].double() - ref).abs() <= ref.abs() * 2.0 ** -8 + 1e-5).all()) and bool((c[:, :, N:] == 5.0).all())
    assert not o.gemm_heads_supported(17, K, K, K, N * K, a.data_ptr(), w.data_ptr()) and not o.gemm_heads_supported(M, K, K, K, N * K, a.data_ptr() + 2, w.data_ptr())
    with pytest.raises(o.KernelError, match="multiple of 32"):
        o.gemm_heads(a.data_ptr(), w.data_ptr(), c.data_ptr(), M, N, K - 8, K, N, 1, K, N * K, N)


def ssd_inputs(H, G, N, P, lens, slots, seed, decays):
    g = torch.Generator().manual_seed(seed)
    T = sum(lens)
    xbc = torch.randn(T, H * P + 2 * G * N, generator=g).bfloat16()
    dtraw = (torch.randn(T, H + 3, generator=g) * 2).bfloat16()
    A_log, bias = {"weak": (torch.full((H,), -4.0), -4.0), "mixed": (torch.linspace(-2, 2, H), -1.0), "strong": (torch.full((H,), 3.0), 2.0)}[decays]
    if decays == "mixed":
        dtraw[::7] += 30.0
    state = torch.randn(max(slots) + 2, H, P, N, generator=g)
    return xbc, dtraw, A_log, torch.full((H,), bias), torch.randn(H, generator=g), state


def ssd_reference(xbc, dtraw, A_log, dt_bias, D, S, H, G, N, P):
    """One row in 64 bits on the device: (y [n, H, P], the state behind it [H, P, N])."""
    n = xbc.shape[0]
    x = xbc[:, :H * P].double().view(n, H, P)
    B, C = (t.double().reshape(n, G, N).repeat_interleave(H // G, dim=1) for t in xbc[:, H * P:].split(G * N, dim=1))
    z = dtraw[:, :H].double() + dt_bias.double()
    dt = torch.where(z > 20, z, torch.log1p(torch.exp(z.clamp(max=20))))
    A, out = torch.exp(A_log.double()), []
    for t in range(n):
        S = torch.exp(-A * dt[t])[:, None, None] * S + x[t][:, :, None] * (dt[t][:, None] * B[t])[:, None, :]
        out.append(torch.einsum("hpn,hn->hp", S, C[t]) + D.double()[:, None] * x[t])
    return torch.stack(out), S


@pytest.mark.parametrize("decays", ["weak", "mixed", "strong"])
@pytest.mark.parametrize("H, G, N, P", [(4, 2, 128, 64), (3, 1, 64, 32), (40, 1, 128, 96)])
def test_state_space_mma(H, G, N, P, decays):
    """Chunks of 64: rows of one token, one beside a chunk's end on either side, several chunks; slots out of order; a slot of no row."""
    o = ops()
    lens, slots = [1, 63, 64, 65, 200], [2, 0, 4, 1, 5]
    starts = [sum(lens[:i]) for i in range(len(lens))]
    xbc, dtraw, A_log, dt_bias, D, state = (t.to(DEV) for t in ssd_inputs(H, G, N, P, lens, slots, H + N, decays))
    st, out = state.clone(), torch.full((sum(lens), H * P), float("nan"), device=DEV)
    assert o.state_space_mma_supported(N, P, xbc.shape[1], xbc.dtype) and not o.state_space_mma_supported(N, P, xbc.shape[1], torch.float32)
    counts = [-(-n // o.state_space_mma_chunk()) for n in lens]
    base = torch.tensor([sum(counts[:i]) for i in range(len(counts))], dtype=torch.int32, device=DEV)
    work = torch.full((sum(counts) * o.state_space_mma_floats(H, G),), float("nan"), device=DEV)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)      # noqa: E731
    o.state_space_mma(xbc, dtraw.data_ptr(), H + 3, A_log, dt_bias, D, st, out, work, base, sum(counts), max(counts), H=H, G=G, N=N, P=P,
                      row_slot=i32(slots), row_q_start=i32(starts), row_q_len=i32(lens))
    for r, n in enumerate(lens):
        s = slice(starts[r], starts[r] + n)
        y, S = ssd_reference(xbc[s], dtraw[s], A_log, dt_bias, D, state[slots[r]].double(), H, G, N, P)
        # the bound of the 32-bit kernels' own test
        assert (out[s].double().view(n, H, P) - y).abs().max() < 1e-5 * y.abs().max(), r
        assert (st[slots[r]].double() - S).abs().max() < 1e-5 * S.abs().max(), r
    assert torch.equal(st[3], state[3]) and torch.equal(st[6], state[6])


def decay_case(lens, slots, H, dk, dv, dtype, decays, seed):
    g = torch.Generator().manual_seed(seed)
    src = (torch.randn(sum(lens), 2 * H * dk + H * dv + 8, generator=g) * 0.8).to(dtype).to(DEV)
    state = (torch.randn(max(slots) + 2, H, dk, dv, generator=g) * 0.3).to(DEV)
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)      # noqa: E731
    rows = dict(row_slot=i32(slots), row_q_start=i32([sum(lens[:i]) for i in range(len(lens))]), row_q_len=i32(lens))
    return src, state, torch.tensor(decays, dtype=torch.float64, device=DEV), rows


def decay_reference(src, S, decays, H, dk, dv):
    """One row in 64 bits: (o [n, H, dv], the state behind it)."""
    x = torch.nn.functional.silu(src.double())
    n = x.shape[0]
    q, k, v = x[:, :H * dk].view(n, H, dk), x[:, H * dk:2 * H * dk].view(n, H, dk), x[:, 2 * H * dk:2 * H * dk + H * dv].view(n, H, dv)
    out = []
    for t in range(n):
        S = decays[:, None, None] * S + k[t][:, :, None] * v[t][:, None, :]
        out.append(torch.einsum("hkv,hk->hv", S, q[t]))
    return torch.stack(out), S


def decay_tiles(o, src, state, decays, rows, lens, H, dk, dv):
    counts = [-(-n // o.decay_attention_tiles_chunk()) for n in lens]
    base = torch.tensor([sum(counts[:i]) for i in range(len(counts))], dtype=torch.int32, device=DEV)
    work = torch.full((sum(counts) * H * o.decay_attention_tiles_floats(dk, dv),), float("nan"), device=DEV)
    out = torch.full((sum(lens), H * dv), float("nan"), device=DEV)
    o.decay_attention_tiles(src, 0, H * dk, 2 * H * dk, decays, state, out, work, base, sum(counts), max(counts), H=H, dk=dk, dv=dv, **rows)
    return out


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("dk, dv", [(128, 128), (64, 64), (128, 64), (64, 128)])
def test_decay_attention_tiles(dk, dv, dtype):
    """Chunks of 64: rows of one token, beside a chunk's end on either side, of more chunks than the scan has under way; decays whose
    powers underflow and close to one; from states that are not zero."""
    o = ops()
    H, lens, slots = 3, [1, 63, 64, 65, 389], [2, 0, 4, 1, 5]
    src, state, decays, rows = decay_case(lens, slots, H, dk, dv, dtype, [0.999, 0.02, 0.7], dk + dv)
    st = state.clone()
    assert o.decay_attention_tiles_supported(dk, dv, src.shape[1], 0, H * dk, 2 * H * dk) and not o.decay_attention_tiles_supported(96, dv, 8, 0, 0, 0)
    out = decay_tiles(o, src, st, decays, rows, lens, H, dk, dv)
    at = 0
    for r, n in enumerate(lens):
        y, S = decay_reference(src[at:at + n], state[slots[r]].double(), decays, H, dk, dv)
        # the bound of the chunked kernels' own test
        assert (out[at:at + n].double().view(n, H, dv) - y).abs().max() < 2e-5 * y.abs().max(), r
        assert (st[slots[r]].double() - S).abs().max() < 2e-5 * S.abs().max(), r
        at += n
    assert torch.equal(st[3], state[3]) and torch.equal(st[6], state[6])


def test_decay_attention_tiles_keep_later_tokens_out():
    """An infinite value reaches its own token's group of four and what lies behind it, nothing before."""
    o = ops()
    lens, H = [100], 2
    src, state, decays, rows = decay_case(lens, [0], H, 128, 128, torch.bfloat16, [0.9, 0.5], 3)
    clean = decay_tiles(o, src, state.clone(), decays, rows, lens, H, 128, 128)
    src[30, 2 * H * 128 + 5] = math.inf
    out = decay_tiles(o, src, state.clone(), decays, rows, lens, H, 128, 128)
    assert torch.equal(out[:28], clean[:28]) and not bool(torch.isfinite(out[30:, 5]).any())


@pytest.mark.parametrize("M, N, K", [(700, 22016, 264), (129, 8, 64), (257, 136, 72), (5000, 264, 64), (1300, 4104, 520)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_gemm_rows_tc_pieces(M, N, K, dtype):
    """More pieces than both accumulators of every SM, a single piece, rows and columns beside a piece's edge, K that ends inside a box."""
    o = ops()
    torch.manual_seed(M + N)
    err = o.new_error_record(DEV)
    x, w = torch.randn(M, K, device=DEV).bfloat16(), (torch.randn(N, K, device=DEV) * 0.1).bfloat16()
    out = torch.full((M + 2, N), 9.0, dtype=dtype, device=DEV)
    o.gemm_tc(x, w, out[:M], err=err)
    o.raise_if_error(err)
    ref = x.double() @ w.double().T
    # products are exact in 32 bit; a sum of K of them, rounded at every step, and one rounding to bfloat16
    bound = K * 2.0 ** -23 * (x.double().abs() @ w.double().abs().T) + (ref.abs() * 2.0 ** -8 if dtype == torch.bfloat16 else 0.0)
    assert bool(((out[:M].double() - ref).abs() <= bound + 1e-6).all()) and bool((out[M:] == 9.0).all())


@pytest.mark.parametrize("scoring, correction, groups", [("softmax", False, None), ("sigmoid", True, (4, 2)), ("softmax_all", True, (4, 2)), ("sigmoid", False, None)])
@pytest.mark.parametrize("T, rows, E, d", [(128, 17, 16, 64), (201, 20, 20, 2048), (2048, 16, 16, 1024), (130, 72, 64, 96), (901, 17, 16, 64), (1003, 72, 64, 96)])
def test_router_of_many_tokens(T, rows, E, d, scoring, correction, groups):
    """Tiles of 16 tokens and 32 rows, the last ones partly filled; blocks of 32 entries that not every warp has."""
    o = ops()
    torch.manual_seed(T + rows)
    x, w = torch.randn(T, d, device=DEV).bfloat16(), (torch.randn(rows, d, device=DEV) * 0.05).bfloat16()
    cor = torch.rand(E, device=DEV) * 0.1 if correction else None
    top = 4
    z = torch.full((T + 1, rows), 9.0, device=DEV)
    choice, weight = torch.full((T, top), -5, dtype=torch.int32, device=DEV), torch.empty(T, top, device=DEV)
    o.router(x, w, E, top, z[:T], choice, weight, scoring=scoring, correction=cor, scale=1.5, normalize=True, groups=groups)
    ref = x.double() @ w.double().T
    # exact products; their sum in 32 bit, rounded at every one of d steps at most
    assert bool(((z[:T].double() - ref).abs() <= 2.0 ** -23 * d * (x.double().abs() @ w.double().abs().T) / 8 + 1e-7).all()) and bool((z[T] == 9.0).all())
    assert (z[:T].double() - ref).norm() < 3e-7 * ref.norm()
    # the same tokens one at a time: another kernel, the same choice wherever the scores are not a rounding apart
    for t in range(0, T, 37):
        z1, c1, w1 = torch.empty(1, rows, device=DEV), torch.empty(1, top, dtype=torch.int32, device=DEV), torch.empty(1, top, device=DEV)
        o.router(x[t:t + 1].contiguous(), w, E, top, z1, c1, w1, scoring=scoring, correction=cor, scale=1.5, normalize=True, groups=groups)
        assert torch.allclose(z1[0], z[t], atol=2e-6, rtol=2e-6) and torch.equal(c1[0], choice[t]) and torch.allclose(w1[0], weight[t], atol=1e-5, rtol=1e-5)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H, KV, dk, dv", [(16, 4, 128, 128), (3, 1, 64, 24), (5, 5, 8, 8), (4, 0, 32, 16), (2, 1, 256, 256)])
@pytest.mark.parametrize("norm, rot, interleaved, unit, from_key, bias", [("whole", 0, False, False, False, True), ("head", 32, False, False, False, True),
                                                                          (None, 16, True, True, True, False), (None, 8, True, False, False, False),
                                                                          ("head", 16, False, True, True, True)])
def test_rows_append_unit_wide_accesses(H, KV, dk, dv, dtype, norm, rot, interleaved, unit, from_key, bias):
    """Rows that begin on 16-byte boundaries beside the same rows one element off, which the narrow kernel takes."""
    o = ops()
    if rot > dk or (from_key and dv > dk) or (rot and not interleaved and rot % 16):
        pytest.skip("no such head")
    g = torch.Generator().manual_seed(H * dk + dv)
    T, ps = 37, 8
    cols = (H + KV) * dk + (0 if from_key else KV * dv)
    data = torch.randn(T, cols, generator=g).to(dtype)
    f = lambda *s: torch.randn(*s, generator=g).to(DEV)      # noqa: E731
    b = f((H + KV) * dk + (0 if from_key else KV * dv)) * 0.1 if bias else None
    qn, kn = (f(H * dk if norm == "whole" else dk), f(max(KV, 1) * dk if norm == "whole" else dk) if KV else None) if norm else (None, None)
    table = f(T, rot // 2, 2) if rot else None
    i32 = lambda v: torch.tensor(v, dtype=torch.int32, device=DEV)      # noqa: E731
    pos, row, bt = i32(list(range(T))), i32([0] * T), i32([[4, 2, 0, 1, 3]])
    got = []
    for pad in (8, 9):
        src = torch.zeros(T, cols + pad, dtype=dtype)
        src[:, :cols] = data
        src = src.to(DEV)
        cache = torch.zeros(5, KV, ps, dk + dv, dtype=dtype, device=DEV) if KV else None
        err = o.new_error_record(DEV)
        o.rows_append_unit(src, pos, row, bt, cache, H=H, KV=KV, dk=dk, dv=dv, ps=ps, row_width=dk + dv, k_off=0, v_off=dk, table=table, rot_dims=rot,
                           interleaved=interleaved, unit_eps=1e-5 if unit else None, value_from_key=from_key, bias=b, q_norm=qn, k_norm=kn,
                           pre_eps=1e-5, norm_whole=norm == "whole", q_temp=(0.3, 5), err=err)
        o.raise_if_error(err)
        got.append((src[:, :cols].double(), cache.double() if KV else torch.zeros(1)))
    tol = 2e-6 if dtype == torch.float32 else 2.0 ** -8      # sums of squares in another order; in bfloat16 the last bit of the one rounding
    for a, c in zip(*got):
        assert (a - c).abs().max() <= tol * c.abs().max().clamp(min=1.0)


@pytest.mark.parametrize("T", [1, 8, 9, 16, 17, 32, 70])
@pytest.mark.parametrize("E, top, F, d", [(16, 4, 64, 256), (3, 2, 40, 72), (5, 5, 1056, 1032)])
@pytest.mark.parametrize("act", ["gated", "relu_squared"])
def test_experts_stream(T, E, top, F, d, act):
    """The stream over the experts' weights beside the tiles of 64 rows on the same routing: rows beside a tile of eight, K and columns beside a
    chunk and a block, an expert that nobody chooses, more rows than a round (T = 70 told as 32), weights on the inputs."""
    o = ops()
    g = torch.Generator().manual_seed(T + F)
    x = torch.randn(T, d, generator=g).bfloat16().to(DEV)
    w1 = (torch.randn(E, (2 if act == "gated" else 1) * F, d, generator=g) / d ** 0.5).bfloat16().to(DEV)
    w2 = (torch.randn(E, d, F, generator=g) / F ** 0.5).bfloat16().to(DEV)
    z = torch.randn(T, E, generator=g)
    if E > top:
        z[:, 1] -= 100.0
    choice, weight = torch.empty(T, top, dtype=torch.int32, device=DEV), torch.empty(T, top, device=DEV)
    o.router_topk(z.to(DEV), E, top, choice, weight)
    tile = o.experts_tile_rows()
    cap = -(-(T * top + (tile - 1) * min(E, T * top)) // tile) * tile
    ss, te = torch.empty(cap, dtype=torch.int32, device=DEV), torch.empty(cap // tile, dtype=torch.int32, device=DEV)
    o.experts_align(choice, E, ss, te, tile)
    scale = (torch.rand(T * top, generator=g) + 0.5).to(DEV) if act == "gated" else None
    got = []
    for stream in (False, True):
        y, zs = torch.zeros(cap, F, dtype=torch.bfloat16, device=DEV), torch.full((T * top, d), float("nan"), device=DEV)
        kw = dict(top=top, act=act, limit=0.9, row_scale=scale)
        if stream:
            o.experts_stream(x, w1, y, ss, te, n=F, k=d, most=min(T, 32), **kw)
            o.experts_stream(y, w2, zs, ss, te, top=top, n=d, k=F, most=min(T, 32))
        else:
            o.experts_gemm(x, w1, y, ss, te, n=F, k=d, **kw)
            o.experts_gemm(y, w2, zs, ss, te, top=top, n=d, k=F)
        got.append((y.float(), zs))
    # the same products in another order of the sums: the last bit of a bfloat16 in between, 2^-8 of a few entries' share
    assert (got[0][0] - got[1][0]).abs().max() <= 2.0 ** -7 * got[0][0].abs().max()
    assert bool(torch.isfinite(got[1][1]).all()) and (got[0][1] - got[1][1]).abs().max() <= 1e-2 * got[0][1].abs().max()


@pytest.mark.parametrize("T, rows, E, d", [(1, 17, 16, 2048), (8, 20, 20, 1000), (127, 40, 33, 4096), (384, 32, 32, 2056)])
def test_router_of_few_tokens(T, rows, E, d):
    o = ops()
    torch.manual_seed(T + rows)
    x, w = torch.randn(T, d, device=DEV).bfloat16(), (torch.randn(rows, d, device=DEV) * 0.05).bfloat16()
    z, choice, weight = torch.empty(T, rows, device=DEV), torch.empty(T, 4, dtype=torch.int32, device=DEV), torch.empty(T, 4, device=DEV)
    o.router(x, w, E, 4, z, choice, weight)
    ref = x.double() @ w.double().T
    assert (z.double() - ref).norm() < 3e-7 * ref.norm()      # exact products, sums of 32 bit
    val, idx = torch.topk(z[:, :E], 4, dim=-1)
    assert torch.equal(choice.long(), idx) and torch.allclose(weight, torch.softmax(val, -1), atol=1e-6)


# slices of 32 value columns once all rows together have more slices of 16 than the chip has SMs; an odd number of slices keeps 16
@pytest.mark.parametrize("H, dk, dv", [(16, 128, 128), (30, 100, 50), (24, 40, 72)])
def test_delta_walk_slices(H, dk, dv):
    """Rows together and one by one: the same bits whatever the slices; both against the kernel that takes the tokens in turn."""
    o = ops()
    g = torch.Generator(device=DEV).manual_seed(H + dk)
    rand = lambda *shape: torch.randn(shape, device=DEV, generator=g)      # noqa: E731
    i32 = lambda x: torch.tensor(x, dtype=torch.int32, device=DEV)      # noqa: E731
    lens, slots = [97, 32, 1], [3, 0, 2]
    T, C = sum(lens), o.delta_rule_chunk()
    qkv, b, a = rand(T, 2 * H * dk + H * dv).bfloat16(), rand(T, H).bfloat16(), rand(T, H * dk)
    A_log, dt_bias, state = rand(H) * 0.5 - 1.0, rand(H * dk), rand(4, H, dv, dk)
    def run(rows, st, out, turns):
        args = (qkv, H * dk, 2 * H * dk, b.data_ptr(), H, a, A_log, dt_bias, st, out)
        where = dict(row_slot=i32([slots[r] for r in rows]), row_q_start=i32([sum(lens[:r]) for r in rows]), row_q_len=i32([lens[r] for r in rows]))
        sizes = dict(H=H, G=H, dk=dk, dv=dv, q_scale=0.3, guard=1e-6)
        if turns:
            return o.delta_rule(*args, **sizes, **where)
        chunks = [-(-lens[r] // C) for r in rows]
        work = torch.full((sum(chunks) * H * o.delta_rule_chunk_floats(dk, dv),), float("nan"), device=DEV)
        o.delta_rule_chunked(*args, work, i32([sum(chunks[:k]) for k in range(len(rows))]), max(chunks), **sizes, **where)
    results = []
    for calls, turns in (([[0, 1, 2]], False), ([[0], [1], [2]], False), ([[0, 1, 2]], True)):
        st, out = state.clone(), torch.full((T, H * dv), float("nan"), device=DEV)
        for rows in calls:
            run(rows, st, out, turns)
        results.append((out, st))
    for x, y, z in zip(*results):
        assert torch.equal(x, y)
        assert (x - z).abs().max() <= 2e-5 * z.abs().max()      # each of the two kernels' own tests allows 1e-5


def decay_tc(o, src, state, decays, rows, lens, H):
    counts = [-(-n // o.decay_attention_tc_chunk()) for n in lens]
    base = torch.tensor([sum(counts[:i]) for i in range(len(counts))], dtype=torch.int32, device=DEV)
    work = torch.full((sum(counts) * H * 128 * 128,), float("nan"), device=DEV)
    out = torch.full((sum(lens) + 1, H * 128), 7.0, device=DEV)
    err = o.new_error_record(DEV)
    o.decay_attention_tc(src, 0, H * 128, 2 * H * 128, decays, state, out, work, base, max(counts), H=H, dk=128, dv=128, err=err, **rows)
    o.raise_if_error(err)
    assert bool((out[-1] == 7.0).all())
    return out[:-1]


@pytest.mark.parametrize("decays", [[0.999, 0.02, 0.7], [0.9995, 0.97, 0.99]])
def test_decay_attention_tc(decays):
    """Chunks of 128: rows of one token, beside a chunk's end on either side, of more chunks than the scan has under way; a slot of no row."""
    o = ops()
    H, lens, slots = 3, [1, 127, 128, 129, 700], [2, 0, 4, 1, 5]
    src, state, dec, rows = decay_case(lens, slots, H, 128, 128, torch.bfloat16, decays, 3)
    st = state.clone()
    assert o.decay_attention_tc_supported(128, 128, src.shape[1], 0, H * 128, 2 * H * 128, src.dtype)
    out = decay_tc(o, src, st, dec, rows, lens, H)
    at = 0
    for r, n in enumerate(lens):
        y, S = decay_reference(src[at:at + n], state[slots[r]].double(), dec, H, 128, 128)
        # three activations of 2^-23 at most each, and sums of 128 terms that are cut off at eight places
        assert (out[at:at + n].double() - y.reshape(n, -1)).norm() < 5e-7 * y.norm(), r
        assert (st[slots[r]].double() - S).norm() < 5e-7 * S.norm(), r
        at += n
    assert torch.equal(st[3], state[3]) and torch.equal(st[6], state[6])


@pytest.mark.parametrize("what", ["q", "k", "v", "state", "small"])
def test_decay_attention_tc_numbers_out_of_the_parts_reach(what):
    """Infinite entries: the chunk that holds them is summed by FMA, and nothing before an infinite token sees it; rows of very small ones."""
    o = ops()
    H, lens, slots = 2, [300], [1]
    src, state, dec, rows = decay_case(lens, slots, H, 128, 128, torch.bfloat16, [0.99, 0.9], 4)
    if what == "state":
        state[1, 0, 3, 5] = float("inf")
    elif what == "small":
        src[140, :256] = 1e-35
    else:
        src[140, {"q": 0, "k": 256, "v": 512}[what] + 7] = float("inf")
    st, ref = state.clone(), state.clone()
    out = decay_tc(o, src, st, dec, rows, lens, H)
    want = decay_tiles(o, src, ref, dec, rows, lens, H, 128, 128)
    assert torch.equal(out[:140].isfinite(), want[:140].isfinite())
    if what in "qkv":
        assert bool(out[:140].isfinite().all()) and not bool(out[140].isfinite().all()) and bool(out[140:, 128:].isfinite().all())
    for a, b in ((out, want), (st, ref)):
        both = a.isfinite() & b.isfinite()
        assert (a[both] - b[both]).norm() < 1e-6 * b[both].norm()


@pytest.mark.parametrize("scaled", [False, True])
@pytest.mark.parametrize("capacity, K, top", [(1, 8, 1), (3, 1032, 2), (4, 2048, 4), (5, 2056, 3), (9, 4096, 8), (130, 24, 4)])
def test_experts_gather_places_beside_a_block(capacity, K, top, scaled):
    """Four places a block: one place, a block's worth, one more, the last block not full; empty places among them and behind them."""
    o = ops()
    torch.manual_seed(capacity + K)
    tokens = (capacity + top - 1) // top + 1
    x = torch.randn(tokens, K, device=DEV).bfloat16()
    places = torch.randint(-1, tokens * top, (capacity,), device=DEV, dtype=torch.int32)
    places[-1] = -1 if capacity > 1 else tokens * top - 1
    scale = torch.rand(tokens * top, device=DEV) if scaled else None
    rows = torch.full((capacity + 1, K), 3.0, dtype=torch.bfloat16, device=DEV)
    o.experts_gather(x, places, top, rows[:capacity], row_scale=scale)
    at = places.long().clamp(min=0)
    want = x[at // top]
    if scaled:
        want = (want.float() * scale[at][:, None]).bfloat16()      # one product, rounded once
    want[places < 0] = 0
    assert torch.equal(rows[:capacity], want) and bool((rows[capacity] == 3.0).all())


@pytest.mark.parametrize("kind", ["normal", "one large entry", "one entry", "positive", "small", "small state"])
def test_decay_attention_tc_is_no_further_off_than_multiply_adds(kind):
    """Rows that one entry dominates, operands of one sign, numbers whose products come near the smallest exponents: errors against 64 bits, beside the kernel that
    sums by FMA in chunks of 64."""
    o = ops()
    H, lens, slots = 2, [389], [1]
    src, state, dec, rows = decay_case(lens, slots, H, 128, 128, torch.bfloat16, [0.999, 0.97], 8)
    g = torch.Generator(device=DEV).manual_seed(9)
    n, C = lens[0], H * 128
    far = torch.rand(n, 2 * H, 128, device=DEV, generator=g)
    if kind == "one large entry":
        src[:, :2 * C] = torch.where(far == far.amax(-1, keepdim=True), 1000.0, src[:, :2 * C].view(n, 2 * H, 128).float()).view(n, -1).bfloat16()
    elif kind == "one entry":
        src[:, :2 * C] *= (far == far.amax(-1, keepdim=True)).view(n, -1)
        src[:, 2 * C:3 * C] *= 8.0
    elif kind == "positive":
        src[:, :3 * C] = src[:, :3 * C].abs() + 1.0
    elif kind == "small":
        src[:, :2 * C] *= 2.0 ** -57
        state.zero_()
    elif kind == "small state":
        src[:, C:2 * C] *= 2.0 ** -118
        state *= 2.0 ** -118
    want, S = decay_reference(src, state[1].double(), dec, H, 128, 128)
    want = want.reshape(n, -1)
    st, ref = state.clone(), state.clone()
    out, fma = decay_tc(o, src, st, dec, rows, lens, H), decay_tiles(o, src, ref, dec, rows, lens, H, 128, 128)
    e, p, es, ps = ((a.double() - b).norm() / b.norm() for a, b in ((out, want), (fma, want), (st[1], S), (ref[1], S)))
    print(f"{kind}: outputs {e:.3g} against {p:.3g}, states {es:.3g} against {ps:.3g}")
    # two activations rounded alike on either side; products left out of a term: 2^-24 of it at most
    assert e <= max(1.05 * p, 1e-7) and es <= max(1.05 * ps, 1e-7)
