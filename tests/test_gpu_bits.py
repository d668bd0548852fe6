"""What a kernel must not let into a result: how a prompt was cut, what shares its step, what lies beside what it reads; and results at the
ends of the number range."""
import math

import pytest
import torch

from test_gpu_kernels import DEV, PagedCase, i32, ops

pytestmark = pytest.mark.gpu


# ------------------------------------------------------------------ 32-bit attention: one order of the sums, whichever kernel takes a token

@pytest.mark.parametrize("H, KV, hd, ps", [(4, 2, 128, 16), (3, 3, 64, 8), (8, 1, 32, 64), (2, 1, 128, 128)])
def test_attention_f32_has_the_bits_of_the_plain_kernel(H, KV, hd, ps):
    """Passes of 128 keys: one key beside a pass' and a tile's ends on either side, one pass and several, portions of one token and of many."""
    o = ops()
    case = PagedCase(torch.float32, H, KV, hd, ps, seq_lens=[2, 33, 127, 128, 129, 160, 161, 257, 400, 700], q_lens=[2, 33, 2, 128, 129, 1, 31, 130, 400, 3],
                     seed=H + hd)
    out, lse = torch.full((case.T, H * hd), 9.0, device=DEV), torch.empty(case.T, H, device=DEV)
    want, want_lse = torch.full_like(out, 9.0), torch.empty_like(lse)
    o.attention_f32(case.params(out, lse=lse), max(case.q_lens))
    o.attention_plain(case.params(want, lse=want_lse))
    assert torch.equal(out, want) and torch.equal(lse, want_lse)


@pytest.mark.parametrize("q_len", [2, 15, 16, 17, 31, 48, 49])
def test_attention_f32_tiles_of_16_queries_have_the_bits_of_the_plain_kernel(q_len):
    """A query beside a tile's end on either side, behind no key, one key, nearly a tile of keys and several passes of them."""
    o = ops()
    starts = [0, 1, 31, 300, 500]
    case = PagedCase(torch.float32, 5, 5, 64, 8, seq_lens=[s + q_len for s in starts], q_lens=[q_len] * 5, seed=q_len)
    out, want = torch.full((case.T, 5 * 64), 9.0, device=DEV), torch.full((case.T, 5 * 64), 9.0, device=DEV)
    o.attention_f32(case.params(out), q_len)
    o.attention_plain(case.params(want))
    assert torch.equal(out, want)


def test_attention_f32_infinite_scores_have_the_bits_of_the_plain_kernel():
    """Keys whose score is minus infinity weigh nothing: a whole pass of them, a part of one, and the first pass."""
    o = ops()
    case = PagedCase(torch.float32, 2, 1, 64, 16, seq_lens=[420], q_lens=[300], seed=8)
    q = case.qcat.view(-1, 2, 64)
    q[:, :, 5] = q[:, :, 5].abs() + 0.1
    for at in list(range(0, 128)) + list(range(250, 400)):
        page = int(case.bt[0, at // 16])
        case.kv[page, 0, 0, at % 16, 5] = -math.inf
    out, want = torch.empty(300, 128, device=DEV), torch.empty(300, 128, device=DEV)
    o.attention_f32(case.params(out), 300)
    o.attention_plain(case.params(want))
    assert torch.equal(out, want) and bool(torch.isfinite(out[100:]).all())


@pytest.mark.parametrize("cuts", [(300,), (299, 1), (1, 299), (31, 269), (33, 129, 138), (128, 128, 44), (2, 1, 297)])
def test_f32_logits_do_not_depend_on_the_cuts(cuts):
    """A 32-bit prompt in portions of any lengths, single tokens among them: the bits of the whole prompt's logits."""
    import helpers
    from delta_b200.config import EngineConfig
    from delta_b200.engine.step import ModelRunner, RowInput
    cfg = helpers.tiny_config("D")
    tokens = helpers.random_tokens(300, cfg["vocab_size"], 4)

    def logits(parts):
        runner = ModelRunner(config_json=cfg, seed=3, engine_config=EngineConfig(max_batch=1, max_seq_len=320, dtype="float32"))
        slot = runner.cache.acquire_slot()
        runner.cache.grow(slot, 300)
        at, got = 0, []
        for n in parts:
            got.append(runner.step([RowInput(slot, tokens[at:at + n], at, list(range(n)))]).clone())
            at += n
        return torch.cat(got)
    assert torch.equal(logits(cuts), logits((300,)))

# ------------------------------------------------------------------ the router: a token's logits are the same in every step

@pytest.mark.parametrize("d, rows, E", [(2048, 17, 16), (2048, 32, 32), (1024, 17, 16), (4096, 65, 64), (520, 20, 20), (2048, 129, 128), (99, 7, 6)])
def test_a_tokens_logits_do_not_depend_on_the_step(d, rows, E):
    """One token, a decode step, portions on either side of every line between the kernels: the same bits for the same token."""
    o = ops()
    g = torch.Generator(device=DEV).manual_seed(d + rows)
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    x = torch.randn(2048, d, device=DEV, generator=g).bfloat16()
    w = (torch.randn(rows, d, device=DEV, generator=g) * 0.05).bfloat16()
    cor = torch.rand(E, device=DEV, generator=g) * 0.1

    def run(T, **kw):
        z, c, wt = torch.empty(T, rows, device=DEV), torch.empty(T, 4, dtype=torch.int32, device=DEV), torch.empty(T, 4, device=DEV)
        o.router(x[:T], w, E, 4, z, c, wt, **kw)
        return z, c, wt
    for kw in (dict(), dict(scoring="sigmoid", correction=cor, scale=2.5, normalize=True)):
        z, c, wt = run(2048, **kw)
        for T in (1, 8, 9, 32, 130, 384, 385, 6 * sms - 1, 6 * sms, 1500):
            zt, ct, wtt = run(T, **kw)
            assert torch.equal(zt, z[:T]) and torch.equal(ct, c[:T]) and torch.equal(wtt, wt[:T]), T
    ref = x.double() @ w.double().T
    assert (z.double() - ref).norm() < 3e-7 * ref.norm()


def test_close_router_scores_are_ranked_by_the_stored_logits():
    """Logits that lie a few units of their last place apart: the choice is the top of what the same call stored, the lowest expert among equals."""
    o = ops()
    d, E = 2048, 16
    g = torch.Generator(device=DEV).manual_seed(5)
    base = torch.randn(d, device=DEV, generator=g)
    w = base.bfloat16().repeat(E, 1)
    w[torch.arange(E, device=DEV), torch.randint(0, d, (E,), device=DEV, generator=g)] += 2.0 ** -6      # one entry of each differs a little
    w[7] = w[3]
    for T in (1, 8, 300, 600, 1200):
        x = torch.randn(T, d, device=DEV, generator=g).bfloat16()
        z, c, wt = torch.empty(T, E, device=DEV), torch.empty(T, 4, dtype=torch.int32, device=DEV), torch.empty(T, 4, device=DEV)
        o.router(x, w, E, 4, z, c, wt)
        want = [[e for _, e in sorted((-v, e) for e, v in enumerate(row))[:4]] for row in z.tolist()]
        assert c.tolist() == want and torch.equal(z[:, 3], z[:, 7])
# ------------------------------------------------------------------ tcgen05 attention over rows: what nobody sees

class RowsCase:
    """Prompt portions over a paged cache of rows (the value behind its key, or the key's front part).  Every row of the cache that no query of
    the step sees is NaN: what another request left in its pages, and the tokens before a window."""

    def __init__(self, H, KV, dk, dv, latent, lens, before, ps, window=0, chunk=0, shaped=False, seed=0, rest=math.nan):
        g = torch.Generator().manual_seed(seed)
        self.H, self.dk, self.dv, self.lens = H, dk, dv, lens
        width = dk if latent else dk + dv
        pages = [-(-(b + n) // ps) for b, n in zip(before, lens)]
        bt = torch.full((len(lens), max(pages)), -1, dtype=torch.int32)
        order = torch.randperm(sum(pages) + 2, generator=g).to(torch.int32)
        cache = torch.full((sum(pages) + 2, KV, ps, width), rest).bfloat16()
        for r, (b, n) in enumerate(zip(before, lens)):
            bt[r, :pages[r]] = order[sum(pages[:r]):sum(pages[:r + 1])]
            low = max(0, b - window + 1) if window else 0
            low = max(low, b // chunk * chunk) if chunk else low
            for at in range(low, b + n):
                cache[bt[r, at // ps], :, at % ps] = torch.randn(KV, width, generator=g).bfloat16()
        T = sum(lens)
        self.q = torch.randn(T, H * dk, generator=g).bfloat16().to(DEV)
        self.cache = cache.to(DEV)
        self.kw = dict(q_stride=H * dk, q_head_stride=dk, H=H, KV=KV, dk=dk, dv=dv, ps=ps, row_width=width, k_off=0, v_off=0 if latent else dk, scale=0.1,
                       window=window, chunk=chunk, block_table=bt.to(DEV), tok_row=i32([r for r, n in enumerate(lens) for _ in range(n)]),
                       tok_pos=i32([b + j for b, n in zip(before, lens) for j in range(n)]), row_q_start=i32([sum(lens[:r]) for r in range(len(lens))]),
                       row_q_len=i32(lens), row_pos_start=i32(before))
        if shaped:
            self.kw.update(softcap=20.0, dist_bias=torch.randn(H, 101, generator=g).to(DEV))

    def run(self, kernel, dtype=torch.bfloat16, q=None):
        o = ops()
        q = (self.q if q is None else q).to(dtype)
        out = torch.full((sum(self.lens), self.H * self.dv), 7.0, dtype=dtype, device=DEV)
        err = o.new_error_record(DEV)
        params = o.row_attn_params(q=q, cache=self.cache.to(dtype), out=out, err=err, **self.kw)
        if kernel == "plain":
            o.attention_rows_plain(params)
        else:
            assert getattr(o, kernel + "_supported")(params)
            getattr(o, kernel)(params, max(self.lens))
        o.raise_if_error(err)
        return out


ROWS_KERNELS = [("attention_rows_wide", (4, 1, 320, 256), True, False), ("attention_rows_wide", (3, 1, 136, 72), True, False),
                ("attention_rows_tc", (4, 2, 128, 128), False, True), ("attention_rows_tc", (4, 2, 72, 104), False, True),
                ("attention_rows_tc", (2, 1, 128, 64), False, False)]


@pytest.mark.parametrize("kernel, shape, latent, shaped", ROWS_KERNELS)
@pytest.mark.parametrize("window, chunk", [(0, 0), (33, 0), (150, 0), (0, 100)])
def test_what_lies_in_rows_that_nobody_sees_does_not_matter(kernel, shape, latent, shaped, window, chunk):
    """A weight of zero times NaN is NaN: the rows behind a portion's last token (one to many of its last tile) and before its first key must
    not meet the product with the values."""
    args = (*shape, latent, [130, 64, 300, 127], [0, 201, 500, 257], 16, window, chunk, shaped)
    case, clean = RowsCase(*args), RowsCase(*args, rest=0.0)
    got, want = case.run(kernel), clean.run("plain", torch.float32)
    assert bool(torch.isfinite(got).all()) and torch.equal(got, clean.run(kernel))
    # weights to 16 bits, one rounding of the output to bfloat16
    assert (got.double() - want.double()).abs().max() < 2.0 ** -8 * want.abs().max()


@pytest.mark.parametrize("kernel, shape, latent, shaped", [k for k in ROWS_KERNELS if k[1][2] % 64])
def test_a_heads_queries_do_not_reach_its_neighbour(kernel, shape, latent, shaped):
    """Heads whose size is no multiple of a box of 64 columns: infinite queries of one head leave the others' bits alone."""
    case = RowsCase(*shape, latent, [130, 70], [0, 100], 16, 0, 0, shaped)
    clean = case.run(kernel).view(200, shape[0], shape[3])
    q = case.q.clone()
    q.view(200, shape[0], shape[2])[50:90, 1] = math.inf
    got = case.run(kernel, q=q).view(200, shape[0], shape[3])
    others = [h for h in range(shape[0]) if h != 1]
    assert torch.equal(got[:, others], clean[:, others]) and torch.equal(got[:50, 1], clean[:50, 1]) and torch.equal(got[90:, 1], clean[90:, 1])


# ------------------------------------------------------------------ sums rounded to nearest; the ends of the number range

@pytest.mark.parametrize("M", [1, 9, 16])
@pytest.mark.parametrize("sign", [1.0, -1.0])
def test_gemm_heads_rounds_its_sums_to_nearest(M, sign):
    """A sum that begins between two bfloat16 numbers and grows by three quarters of its last place with every 16 entries: rounded to nearest at
    every step it passes the middle, cut off at every step it stays there and goes to the even neighbour."""
    o = ops()
    K, N = 256, 16
    a, w = torch.zeros(M, K, device=DEV), torch.ones(N, K, device=DEV)
    a[:, 0] = sign
    a[:, 1] = sign * 2.0 ** -8
    for block in range(1, K // 32):      # (the kernel's MMAs take the first and the second half of every eight entries)
        a[:, 32 * block] = sign * 1.5 * 2.0 ** -24
        a[:, 32 * block + 4] = sign * 1.5 * 2.0 ** -24
    a, w = a.bfloat16(), w.bfloat16()
    c = torch.empty(M, N, dtype=torch.bfloat16, device=DEV)
    o.gemm_heads(a.data_ptr(), w.data_ptr(), c.data_ptr(), M, N, K, K, N, 1, M * K, N * K, M * N)
    exact = a.double() @ w.double().T
    assert bool((exact.abs() > 1.0 + 2.0 ** -8).all())
    assert torch.equal(c, torch.full_like(c, sign * (1.0 + 2.0 ** -7)))


@pytest.mark.parametrize("value", [math.inf, -math.inf, 3.4e38, -3.4e38, 3.39e38])
def test_state_space_mma_keeps_infinite_and_large_states(value):
    """A state entry that is infinite, or finite and above bfloat16's largest number: it stays in its channel, and the outputs are what 64 bits give."""
    from test_gpu_tiles import ssd_inputs, ssd_reference
    o = ops()
    H, G, N, P, lens = 4, 2, 128, 64, [130]
    xbc, dtraw, A_log, dt_bias, D, state = (t.to(DEV) for t in ssd_inputs(H, G, N, P, lens, [0], 3, "weak"))
    C = xbc[:, H * P + G * N:]
    C.copy_(torch.where(C.abs() < 2.0 ** -3, torch.full_like(C, 0.5), C) * 2.0 ** -10)      # no zeros, and outputs in range
    state[0, 1, 5, 77] = value
    st, out = state.clone(), torch.empty(130, H * P, device=DEV)
    counts = -(-130 // o.state_space_mma_chunk())
    work = torch.empty(counts * o.state_space_mma_floats(H, G), device=DEV)
    o.state_space_mma(xbc, dtraw.data_ptr(), H + 3, A_log, dt_bias, D, st, out, work, i32([0]), counts, counts, H=H, G=G, N=N, P=P, row_slot=i32([0]),
                      row_q_start=i32([0]), row_q_len=i32([130]))
    y, S = ssd_reference(xbc, dtraw, A_log, dt_bias, D, state[0].double(), H, G, N, P)
    y, S, out, st = y.view(130, H * P), S, out.double(), st[0].double()
    inf = torch.isinf(y)
    assert torch.equal(torch.isinf(out), inf) and torch.equal(out[inf], y[inf]) and not bool(torch.isnan(out).any())
    assert bool(((out - y)[~inf].abs() <= 1e-6 * y[~inf].abs().clamp(min=1.0)).all() if math.isinf(value) else ((out - y).abs() <= 1e-5 * y.abs().clamp(min=1.0)).all())
    inf = torch.isinf(S)
    assert torch.equal(torch.isinf(st), inf) and torch.equal(st[inf], S[inf]) and bool(((st - S)[~inf].abs() <= 1e-5 * S[~inf].abs().clamp(min=1.0)).all())


@pytest.mark.parametrize("decays", ["weak", "mixed", "strong"])
@pytest.mark.parametrize("H, G, N, P", [(4, 2, 128, 64), (3, 1, 64, 32)])
def test_state_space_mma_loses_no_part_of_its_operands(H, G, N, P, decays):
    """Several chunks against 64 bits in the 2-norm: sums of 32 bit leave about 1e-7; without the lowest part of an operand it would be 2^-17 and
    with two parts rounded together 2^-20."""
    from test_gpu_tiles import ssd_inputs, ssd_reference
    o = ops()
    n = 700
    xbc, dtraw, A_log, dt_bias, D, state = (t.to(DEV) for t in ssd_inputs(H, G, N, P, [n], [0], N, decays))
    st, out = state.clone(), torch.empty(n, H * P, device=DEV)
    chunks = -(-n // o.state_space_mma_chunk())
    work = torch.empty(chunks * o.state_space_mma_floats(H, G), device=DEV)
    o.state_space_mma(xbc, dtraw.data_ptr(), H + 3, A_log, dt_bias, D, st, out, work, i32([0]), chunks, chunks, H=H, G=G, N=N, P=P, row_slot=i32([0]),
                      row_q_start=i32([0]), row_q_len=i32([n]))
    y, S = ssd_reference(xbc, dtraw, A_log, dt_bias, D, state[0].double(), H, G, N, P)
    assert (out.double() - y.view(n, H * P)).norm() < 3e-7 * y.norm() and (st[0].double() - S).norm() < 3e-7 * S.norm()


@pytest.mark.parametrize("n", [1, 63, 65, 130])
@pytest.mark.parametrize("H, G, N, P", [(4, 2, 128, 64), (3, 1, 64, 32)])
def test_state_space_mma_the_next_rows_tokens_stay_out(H, G, N, P, n):
    """What lies behind a row's last token is another request's: not a number there leaves the row's outputs and state as they are."""
    from test_gpu_tiles import ssd_inputs
    o = ops()
    xbc, dtraw, A_log, dt_bias, D, state = (t.to(DEV) for t in ssd_inputs(H, G, N, P, [n, 70], [0, 1], 5, "mixed"))

    def run(xbc, dtraw):
        st, out = state.clone(), torch.zeros(n + 70, H * P, device=DEV)
        counts = [-(-n // o.state_space_mma_chunk()), 2]
        work = torch.empty(sum(counts) * o.state_space_mma_floats(H, G), device=DEV)
        err = o.new_error_record(DEV)
        o.state_space_mma(xbc, dtraw.data_ptr(), H + 3, A_log, dt_bias, D, st, out, work, i32([0, counts[0]]), sum(counts), max(counts), H=H, G=G, N=N, P=P,
                          row_slot=i32([0, 1]), row_q_start=i32([0, n]), row_q_len=i32([n, 70]), err=err)
        o.raise_if_error(err)
        return out[:n], st[0]
    out, st = run(xbc, dtraw)
    xbc, dtraw = xbc.clone(), dtraw.clone()
    xbc[n:], dtraw[n:] = math.nan, math.nan
    got, got_st = run(xbc, dtraw)
    assert torch.equal(got, out) and torch.equal(got_st, st) and bool(torch.isfinite(out).all())


@pytest.mark.parametrize("M", [65535 * 32 + 1, 65535 * 64])
@pytest.mark.parametrize("dtype, K", [(torch.float32, 4), (torch.float32, 3), (torch.bfloat16, 4)])
def test_gemm_plain_takes_millions_of_rows(M, dtype, K):
    """The most rows that tiles of 64 can number, one more than tiles of 32 can; one row more than that is refused."""
    o = ops()
    a = torch.randint(-3, 4, (M, K), device=DEV).to(dtype)
    w = torch.randint(-3, 4, (2, K), device=DEV).to(dtype)
    out = torch.empty(M, 2, device=DEV)
    o.gemm_nt_plain(a, w, out)
    assert torch.equal(out, (a.float()[:, None, :] * w.float()[None]).sum(-1))
    if M == 65535 * 64:
        a, out = torch.zeros(M + 1, K, dtype=dtype, device=DEV), torch.empty(M + 1, 2, device=DEV)
        with pytest.raises(o.KernelError, match="too large"):
            o.gemm_nt_plain(a, w, out)


# ------------------------------------------------------------------ single tokens whose key tiles are shared by four warps; lists of pieces at their ends

@pytest.mark.parametrize("shape", [(16, 1, 320, 256), (5, 1, 272, 160), (12, 2, 192, 144)])
@pytest.mark.parametrize("splits", [1, 2, 7])
@pytest.mark.parametrize("shaped, window", [(False, 0), (True, 0), (False, 50)])
def test_key_warps_of_single_tokens(shape, splits, shaped, window):
    """Four warps take tiles of 32 keys in turn and meet under one maximum: fewer keys than a tile, tiles for some warps only, one key beside a
    round of all four, more splits than tiles; the largest score with any of the warps."""
    o = ops()
    H, KV, dk, dv = shape
    before = [0, 19, 31, 32, 95, 127, 128, 129, 700, 1100]
    case = RowsCase(H, KV, dk, dv, True, [1] * len(before), before, 16, window, 0, shaped, seed=dk + splits)
    for r, b in enumerate(before):      # a key that stands out, in another warp's tile for every row
        at = max(b - 37 * r, max(0, b - window + 1) if window else 0)
        page = int(case.kw["block_table"][r, at // 16])
        case.cache[page, :, at % 16, :8] += 6.0
    sink, gate = torch.randn(H, device=DEV), torch.randn(len(before), H, device=DEV).bfloat16()

    def run(dtype):
        q, cache = case.q.to(dtype), case.cache.to(dtype)
        g = gate.to(dtype)
        out = torch.full((len(before), H * dv), 7.0, dtype=dtype, device=DEV)
        p = o.row_attn_params(q=q, cache=cache, out=out, sink=sink, gate_ptr=g.data_ptr(), gate_stride=H, **case.kw)
        if dtype == torch.float32:
            o.attention_rows_plain(p)
        else:
            assert o.attention_rows_mma_key_warps(p) == 4
            n = o.attention_rows_mma_scratch_floats(p.T, H, dv, splits)
            scratch = torch.full((max(n, 1),), math.nan, device=DEV)
            o.attention_rows_mma(p, H // KV, splits, scratch if splits > 1 else None)
        torch.cuda.synchronize()
        return out.double()
    got, want = run(torch.bfloat16), run(torch.float32)
    # weights to 16 bits, one rounding of the output to bfloat16 (2^-9 of it)
    assert bool(torch.isfinite(got).all()) and (got - want).abs().max() < 2.0 ** -8 * want.abs().max()


@pytest.mark.parametrize("rows, n", [(256, 2), (257, 2), (128, 129), (511, 1), (512, 2), (600, 3)])
@pytest.mark.parametrize("kernel, shape, latent", [("attention_rows_tc", (2, 1, 64, 64), False), ("attention_rows_wide", (2, 1, 136, 64), True)])
def test_rows_pieces_at_the_ends_of_their_list(kernel, shape, latent, rows, n):
    """As many pairs of row and query tile as the list holds, one more, and more rows than its entries can name: the old numbering takes over."""
    lens = [n] * rows
    lens[rows // 2], lens[rows - 1] = 140 if n == 3 else n, 1 if n == 2 else n
    case = RowsCase(*shape, latent, lens, [(7 * r) % 50 for r in range(rows)], 8, seed=rows)
    got, want = case.run(kernel).double(), case.run("plain", torch.float32).double()
    assert (got - want).abs().max() < 2.0 ** -8 * want.abs().max()


@pytest.mark.parametrize("rows, n, window", [(64, 33, 0), (65, 33, 0), (32, 200, 40), (511, 2, 0), (520, 2, 0), (7, 1100, 0)])
def test_prefill_pieces_at_the_ends_of_their_list(rows, n, window):
    o = ops()
    q_lens = [n if r % 5 else max(1, n - 1) for r in range(rows)]
    case = PagedCase(torch.bfloat16, 2, 1, 64, 16, seq_lens=[q + (11 * r) % 60 for r, q in enumerate(q_lens)], q_lens=q_lens, seed=rows)
    out, want = torch.empty(case.T, 128, dtype=torch.bfloat16, device=DEV), torch.empty(case.T, 128, dtype=torch.bfloat16, device=DEV)
    o.attention_prefill_tc(case.params(out, window=window), max(q_lens))
    o.attention_plain(case.params(want, window=window))
    # both round their output to bfloat16; the weights of the one have 16 bits
    assert (out.double() - want.double()).abs().max() < 2.0 ** -7 * want.double().abs().max()


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("taps", [2, 3, 4])
@pytest.mark.parametrize("C, stride, with_bias, silu", [(8, 8, True, True), (1032, 1040, False, True), (264, 264, True, False)])
def test_convolution_over_tiles_of_eight_tokens(C, stride, with_bias, silu, taps, dtype):
    """Rows that begin and end inside a tile of eight tokens, several in one tile, shorter than the taps; a last tile of one token."""
    o = ops()
    lens, slots = [1, 2, 3, 9, 8, 1, 1, 7, 17], [4, 2, 7, 0, 1, 3, 5, 6, 8]
    g = torch.Generator().manual_seed(C + taps)
    T = sum(lens)
    x = torch.randn(T, stride, generator=g).to(dtype)
    w, b = torch.randn(C, taps, generator=g), torch.randn(C, generator=g) if with_bias else None
    state = torch.randn(10, taps - 1, C, generator=g)
    st, out = state.to(DEV), torch.full((T, C), 9.0, dtype=dtype, device=DEV)
    starts = [sum(lens[:i]) for i in range(len(lens))]
    o.conv_silu(x.to(DEV), stride, w.to(DEV), b.to(DEV) if with_bias else None, st, out, tok_row=i32([r for r, n in enumerate(lens) for _ in range(n)]),
                row_slot=i32(slots), row_q_start=i32(starts), row_q_len=i32(lens), silu=silu)
    for r, n in enumerate(lens):
        seq = torch.cat([state[slots[r]].double(), x[starts[r]:starts[r] + n, :C].double()])
        want = sum(w[:, j].double() * seq[j:j + n] for j in range(taps)) + (b.double() if with_bias else 0.0)
        want = torch.nn.functional.silu(want) if silu else want
        # up to five products of 32 bit, and the one rounding of the output
        assert bool(((out[starts[r]:starts[r] + n].double().cpu() - want).abs() <= (2.0 ** -8 if dtype == torch.bfloat16 else 2e-6) * want.abs() + 5e-6).all()), r
        assert torch.equal(st[slots[r]].cpu(), seq[-(taps - 1):].float())
    assert torch.equal(st[9].cpu(), state[9])
