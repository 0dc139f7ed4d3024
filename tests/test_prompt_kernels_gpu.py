"""Kernels of prompt steps at the sizes where they can go wrong: edges of tiles, remainders, later portions, slots
of a page that hold no number."""
import math

import pytest
import torch

import plain_llama as P
from test_kernels_gpu import DEV, PagedCase, close, ops

pytestmark = pytest.mark.gpu


def i32(x):
    return torch.tensor(x, dtype=torch.int32, device=DEV)


def stored(case, dtype, empty):
    """The caches of a ``PagedCase`` with every position up to the lengths filled and the rest ``empty``."""
    kc, vc = torch.full_like(case.k_cache, empty), torch.full_like(case.v_cache, empty)
    for s, L in enumerate(case.lengths):
        for t in range(L):
            pg = int(case.table[s, t // 64])
            kc[pg, :, t % 64], vc[pg, :, t % 64] = case.k[s][t], case.v[s][t]
    return kc.to(dtype).to(DEV), vc.to(dtype).to(DEV)


@pytest.mark.parametrize("m", [63, 64, 65, 129])
@pytest.mark.parametrize("n,k", [(64, 32), (63, 31), (65, 33), (130, 576), (4, 1)])
def test_float32_product_at_the_edges_of_its_tiles(m, n, k):
    o = ops()
    g = torch.Generator().manual_seed(m + 10 * n + 100 * k)
    a, w = torch.randn(m, k, generator=g), torch.randn(n, k, generator=g) / math.sqrt(k)
    bias = torch.randn(n, generator=g)
    want = P.linear(a, w, bias)
    room = torch.full((m * n + 1,), 7.0, device=DEV)
    for off in (0, 1):  # (a destination that is not 16-byte aligned)
        out = room[off:off + m * n].view(m, n)
        o.gemm_simt(a.to(DEV), w.to(DEV), bias.to(DEV), out, o.STORE)
        close(out, want, "float32", f"store at {off}")
        o.gemm_simt(a.to(DEV), w.to(DEV), None, out, o.ADD_F32)
        close(out, want + P.linear(a, w), "float32", f"add at {off}")


@pytest.mark.parametrize("nq,nkv,d", [(3, 3, 64), (6, 2, 48), (4, 1, 128), (2, 2, 4), (3, 1, 100)])
@pytest.mark.parametrize("window", [0, 1, 70])
@pytest.mark.parametrize("splits", [1, 3])
def test_float32_prompt_attention_in_tiles(nq, nkv, d, window, splits):
    """Whole prompts and later portions; a slot that no token has filled holds NaN."""
    o = ops()
    lengths, new = [70, 1, 200, 64, 333, 129], [70, 1, 5, 64, 200, 65]
    case = PagedCase(lengths, new, nq, nkv, d, "float32", seed=d + nq)
    kc, vc = stored(case, torch.float32, math.nan)
    q = case.packed()[2]
    n, stride = q.shape[0], nq * d + 8
    qd = torch.full((n, stride), 3.0, device=DEV)
    qd[:, :nq * d] = q.reshape(n, -1).to(DEV)
    tiles = [[i, q0] for i, c in enumerate(new) for q0 in range(0, c, 64)]
    out = torch.full((n, nq * d), 5.0, device=DEV)
    partial = torch.full((n * nq * splits * (d + 2),), math.nan, device=DEV) if splits > 1 else None
    o.attention_tile_f32(qd, stride, kc, vc, i32(tiles), i32([sum(new[:i]) for i in range(len(new))]),
                         i32([L - c for L, c in zip(lengths, new)]), i32(new), case.table.to(DEV), out, nq, nkv, d,
                         window, 1.0 / math.sqrt(d), splits, partial)
    r = 0
    for s, L in enumerate(lengths):
        full = P.causal_attention(case.q[s], case.k[s], case.v[s], window)
        close(out[r:r + new[s]], full[L - new[s]:].reshape(new[s], -1), "float32", f"sequence {s}")
        r += new[s]


@pytest.mark.parametrize("nq,nkv", [(3, 3), (6, 2), (4, 1)])
@pytest.mark.parametrize("window", [0, 1, 70, 300])
@pytest.mark.parametrize("sms", [1, 40, 1000])
def test_float32_prompt_attention_on_tcgen05(nq, nkv, window, sms):
    """Head size 64, whole prompts and later portions, as the plans for one, some and very many SMs cut them (whole tiles, slices
    of unequal number); a slot that no token has filled holds NaN."""
    o = ops()
    d, lengths, new = 64, [70, 200, 64, 333, 129, 1000], [70, 5, 64, 200, 65, 1000]
    case = PagedCase(lengths, new, nq, nkv, d, "float32", seed=5 * nq + window)
    kc, vc = stored(case, torch.float32, math.nan)
    q = case.packed()[2]
    n, stride = q.shape[0], nq * d + 8
    qd = torch.full((n, stride), 3.0, device=DEV)
    qd[:, :nq * d] = q.reshape(n, -1).to(DEV)
    first, start, count, starts = wide_inputs(new, lengths)
    plan = o.attention_split_f32_plan(new, starts, window, nq, sms)
    if plan is None:  # (a window of one key: the other kernel's; these units run all the same)
        plan = torch.tensor([(i, q0, 0, 1) for i, c in enumerate(new) for q0 in range(0, c, 128)]).numpy(), 1
    units, slices = plan
    out = torch.full((n, nq * d), 5.0, device=DEV)
    partial = torch.full((n * nq * slices * (d + 2),), math.nan, device=DEV) if slices > 1 else None
    o.attention_split_f32(qd, stride, kc, vc, i32(units), first, start, count, case.table.to(DEV), out, nq, nkv, d, window,
                          1.0 / math.sqrt(d), slices, partial)
    o.check_status(DEV)
    r = 0
    for s, L in enumerate(lengths):
        full = P.causal_attention(case.q[s], case.k[s], case.v[s], window)[L - new[s]:].reshape(new[s], -1).double()
        got = out[r:r + new[s]].cpu().double()
        # scores of order one within 2e-7 of themselves, sums of at most 1,000 weights: 1e-6 of the result's 2-norm
        assert float((got - full).norm() / full.norm()) < 1e-6, s
        r += new[s]


def test_float32_prompt_attention_on_tcgen05_with_values_that_are_no_numbers():
    """An infinity or NaN among values or keys is felt by the queries that see it, as the kernel with chains of multiply-adds
    has it, and by no other."""
    o = ops()
    nq, nkv, d, L = 2, 1, 64, 300
    case = PagedCase([L], [L], nq, nkv, d, "float32", seed=3)
    case.v[0][100, 0, 5], case.v[0][200, 0, 40], case.k[0][250, 0, 7] = math.inf, math.nan, math.inf
    kc, vc = stored(case, torch.float32, 0.0)
    q = case.packed()[2].reshape(L, -1).contiguous().to(DEV)
    first, start, count, starts = wide_inputs([L], [L])
    seq, pos = torch.zeros(L, dtype=torch.int32, device=DEV), torch.arange(L, dtype=torch.int32, device=DEV)
    want = torch.empty(L, nq * d, device=DEV)
    o.attention_generic(q, nq * d, kc, vc, pos, seq, case.table.to(DEV), want, nq, nkv, d, 0, 0.125, 1, None)
    assert torch.isnan(want[299]).any() and torch.isinf(want[150]).any() and torch.isfinite(want[:100]).all()
    for units, slices in (([(0, 0, 0, 1), (0, 128, 0, 1), (0, 256, 0, 1)], 1),
                          ([(0, 0, 0, 1), (0, 128, 0, 2), (0, 128, 1, 2), (0, 256, 0, 3), (0, 256, 1, 3), (0, 256, 2, 3)], 3)):
        out = torch.full((L, nq * d), 5.0, device=DEV)
        partial = torch.full((L * nq * slices * (d + 2),), math.nan, device=DEV) if slices > 1 else None
        o.attention_split_f32(q, nq * d, kc, vc, i32(units), first, start, count, case.table.to(DEV), out, nq, nkv, d, 0, 0.125,
                              slices, partial)
        o.check_status(DEV)
        assert torch.equal(torch.isnan(out), torch.isnan(want)) and torch.equal(torch.isinf(out), torch.isinf(want))
        fine = torch.isfinite(want)
        assert torch.allclose(out[fine], want[fine], atol=5e-6)


def wide_inputs(new, lengths):
    starts = [L - c for L, c in zip(lengths, new)]
    return i32([sum(new[:i]) for i in range(len(new))]), i32(starts), i32(new), starts


@pytest.mark.parametrize("nq,nkv", [(4, 1), (2, 2), (6, 3)])
@pytest.mark.parametrize("window", [0, 70, 300])
@pytest.mark.parametrize("pad,sms", [(0, 1000), (24, 1)])
def test_wide_prompt_attention_on_tcgen05(nq, nkv, window, pad, sms):
    """Head size 128: whole prompts and later portions, one tile of queries a CTA and two, more pages than the ring holds."""
    o = ops()
    d, lengths, new = 128, [70, 1, 200, 64, 333, 129, 1500], [70, 1, 5, 64, 200, 65, 1500]
    case = PagedCase(lengths, new, nq, nkv, d, "bfloat16", seed=5 * nq + window)
    kc, vc = stored(case, torch.bfloat16, math.nan)
    q = case.packed()[2]
    n, stride = q.shape[0], nq * d + pad
    qd = torch.full((n, stride), 3.0, dtype=torch.bfloat16, device=DEV)
    qd[:, :nq * d] = q.reshape(n, -1).bfloat16().to(DEV)
    first, start, count, starts = wide_inputs(new, lengths)
    units = o.attention_wide_plan(new, starts, window, nq, sms)
    out = torch.full((n, nq * d), 5.0, dtype=torch.bfloat16, device=DEV)
    o.attention_wide_tc(qd, stride, kc, vc, torch.from_numpy(units).to(DEV), first, start, count, case.table.to(DEV), out,
                        nq, nkv, d, window, 1.0 / math.sqrt(d))
    o.check_status(DEV)
    r = 0
    for s, L in enumerate(lengths):
        full = P.causal_attention(case.q[s], case.k[s], case.v[s], window)
        close(out[r:r + new[s]], full[L - new[s]:].reshape(new[s], -1), "bfloat16", f"sequence {s}")
        r += new[s]


@pytest.mark.parametrize("dim,rot", [(128, 64), (64, 32)])
@pytest.mark.parametrize("heads,sms,sharp", [(1, 1000, 1.0), (3, 1, 1.0), (2, 1, 6.0)])
def test_wide_prompt_attention_over_expanded_latents(dim, rot, heads, sms, sharp):
    """Keys whose last part all heads share; ``sharp`` scores make the running maximum rise from page to page."""
    o = ops()
    g = torch.Generator().manual_seed(dim + heads)
    lengths, new = [64, 1, 200, 333, 1000], [64, 1, 5, 200, 1000]
    first, start, count, starts = wide_inputs(new, lengths)
    pages = [-(-L // 64) for L in lengths]
    rows, base = 64 * sum(pages), [64 * sum(pages[:i]) for i in range(len(pages))]
    n = sum(new)
    q = (torch.randn(n, heads, dim + rot, generator=g) * sharp).bfloat16()
    kv = torch.randn(rows, heads * 2 * dim, generator=g).bfloat16()
    kr = torch.zeros(rows, 64)
    kr[:, :rot] = torch.randn(rows, rot, generator=g)
    kr = kr.bfloat16()
    units = torch.from_numpy(o.attention_wide_plan(new, starts, 0, heads, sms)).to(DEV)
    out = torch.full((n, heads * dim), 5.0, dtype=torch.bfloat16, device=DEV)
    scale = (dim + rot) ** -0.5
    o.attention_wide_tc_expanded(q.reshape(n, -1).to(DEV), kv.to(DEV), kr.to(DEV), units, i32(base), first, start, count,
                                 out, heads, dim, rot, dim, 0, scale)
    o.check_status(DEV)
    r = 0
    for s, L in enumerate(lengths):
        part = slice(base[s], base[s] + L)
        k = torch.cat([kv[part, :heads * dim].view(L, heads, dim), kr[part, None, :rot].expand(L, heads, rot)], -1).double()
        v = kv[part, heads * dim:].view(L, heads, dim).double()
        qs = q[r:r + new[s]].double()
        scores = torch.einsum("thd,shd->hts", qs, k) * scale
        hidden = torch.arange(L)[None, :] > torch.arange(L - new[s], L)[:, None]
        want = torch.einsum("hts,shd->thd", torch.softmax(scores.masked_fill(hidden, -math.inf), -1), v)
        close(out[r:r + new[s]], want.reshape(new[s], -1), "bfloat16", f"sequence {s}")
        r += new[s]


def spoilt(v, at):
    """Values with infinities and NaN in two of their columns at the positions ``at``."""
    v = v.clone()
    for i, t in enumerate(at):
        v[t, :, 5] = math.nan if i % 2 else math.inf
        v[t, :, 50] = -math.inf if i % 2 else math.inf
    return v


def check_spoilt(got, fine, v, at, starts, window, what):
    """``got`` is ``fine`` for the queries that see none of the positions ``at`` and in the columns where these are
    numbers; a query that sees them has what their sum with a positive weight each is."""
    for t in range(got.shape[0]):
        seen = [a for a in at if a <= starts + t and (window == 0 or starts + t - a < window)]
        want = fine[t] + sum((torch.where(torch.isfinite(v[a].double()), 0.0, v[a].double()) for a in seen), torch.zeros(()))
        same = torch.isfinite(want)
        close(got[t][same], want[same], "bfloat16", f"{what}, query {t}")
        assert torch.equal(torch.nan_to_num(got[t][~same].double(), 7.0), torch.nan_to_num(want[~same], 7.0)), (what, t)


@pytest.mark.parametrize("window", [0, 70])
@pytest.mark.parametrize("sms", [1000, 1])
def test_wide_prompt_attention_and_values_that_are_no_numbers(window, sms):
    """An infinity or a NaN among the values is not felt by a query that does not see its token: the ones before it in
    its tile of 128, the ones whose window has passed it."""
    o = ops()
    d, nq, nkv = 128, 4, 2
    lengths, new, at = [70, 300, 700], [70, 300, 500], [[69], [0, 64, 200, 299], [100, 230, 450, 451, 640]]
    case = PagedCase(lengths, new, nq, nkv, d, "bfloat16", seed=window)
    finite = case.v
    case.v = [spoilt(v, a) for v, a in zip(finite, at)]
    kc, vc = stored(case, torch.bfloat16, math.nan)
    q = case.packed()[2]
    n = q.shape[0]
    first, start, count, starts = wide_inputs(new, lengths)
    units = o.attention_wide_plan(new, starts, window, nq, sms)
    out = torch.full((n, nq * d), 5.0, dtype=torch.bfloat16, device=DEV)
    o.attention_wide_tc(q.reshape(n, -1).bfloat16().to(DEV), nq * d, kc, vc, torch.from_numpy(units).to(DEV), first, start,
                        count, case.table.to(DEV), out, nq, nkv, d, window, 1.0 / math.sqrt(d))
    o.check_status(DEV)
    r = 0
    for s, L in enumerate(lengths):
        zeroed = torch.where(torch.isfinite(case.v[s]), case.v[s], torch.zeros(()))
        fine = P.causal_attention(case.q[s], case.k[s], zeroed, window)[L - new[s]:]
        check_spoilt(out[r:r + new[s]].cpu().view(new[s], nq, d), fine, case.v[s].repeat_interleave(nq // nkv, 1), at[s],
                     L - new[s], window, f"sequence {s}")
        r += new[s]


@pytest.mark.parametrize("dim,rot", [(128, 64), (64, 32)])
@pytest.mark.parametrize("sms", [1000, 1])
def test_expanded_latents_and_values_that_are_no_numbers(dim, rot, sms):
    o = ops()
    g = torch.Generator().manual_seed(dim + sms)
    heads, lengths, new, at = 2, [64, 333], [64, 200], [[63], [20, 140, 200, 201, 330]]
    first, start, count, starts = wide_inputs(new, lengths)
    base, rows, n = [0, 64], 64 + 384, sum(new)
    q = torch.randn(n, heads, dim + rot, generator=g).bfloat16()
    kv, kr = torch.randn(rows, heads * 2 * dim, generator=g).bfloat16(), torch.zeros(rows, 64)
    kr[:, :rot] = torch.randn(rows, rot, generator=g)
    kr, v = kr.bfloat16(), kv[:, heads * dim:].view(rows, heads, dim)
    for s in range(2):
        v[base[s]:base[s] + lengths[s]] = spoilt(v[base[s]:base[s] + lengths[s]], at[s])
    v[base[1] + lengths[1]:] = math.nan  # (rows past the sequence's last position)
    units = torch.from_numpy(o.attention_wide_plan(new, starts, 0, heads, sms)).to(DEV)
    out = torch.full((n, heads * dim), 5.0, dtype=torch.bfloat16, device=DEV)
    scale = (dim + rot) ** -0.5
    o.attention_wide_tc_expanded(q.reshape(n, -1).to(DEV), kv.to(DEV), kr.to(DEV), units, i32(base), first, start, count,
                                 out, heads, dim, rot, dim, 0, scale)
    o.check_status(DEV)
    r = 0
    for s, L in enumerate(lengths):
        part = slice(base[s], base[s] + L)
        k = torch.cat([kv[part, :heads * dim].view(L, heads, dim), kr[part, None, :rot].expand(L, heads, rot)], -1).double()
        zeroed = torch.where(torch.isfinite(v[part].double()), v[part].double(), 0.0)
        scores = torch.einsum("thd,shd->hts", q[r:r + new[s]].double(), k) * scale
        hidden = torch.arange(L)[None, :] > torch.arange(L - new[s], L)[:, None]
        fine = torch.einsum("hts,shd->thd", torch.softmax(scores.masked_fill(hidden, -math.inf), -1), zeroed)
        check_spoilt(out[r:r + new[s]].cpu().view(new[s], heads, dim), fine, v[part], at[s], L - new[s], 0, f"sequence {s}")
        r += new[s]


@pytest.mark.parametrize("rank,rot", [(256, 32), (24, 64), (512, 0)])
def test_cached_latent_rows_one_after_another(rank, rot):
    o = ops()
    g = torch.Generator().manual_seed(rank)
    lengths, new = [64, 1, 130], [3, 1, 130]
    cache = torch.randn(9, 1, 64, rank + rot, generator=g).bfloat16()
    table = torch.tensor([[4, -1, -1], [7, -1, -1], [2, 8, 0]], dtype=torch.int32)
    blocks = [(0, 0), (1, 0), (2, 0), (2, 1), (2, 2)]
    c, r = (torch.full((320, w), 9.0, dtype=torch.bfloat16, device=DEV) for w in (rank, 64))
    _, start, count, _ = wide_inputs(new, lengths)
    o.latent_rows(cache.to(DEV), i32(blocks), start, count, table.to(DEV), c, r)
    want = torch.zeros(320, rank + 64, dtype=torch.bfloat16)
    for b, (s, p) in enumerate(blocks):
        rows = min(64, lengths[s] - 64 * p)
        want[64 * b:64 * b + rows, :rank + rot] = cache[int(table[s, p]), 0, :rows]
    assert torch.equal(torch.cat([c, r], 1).cpu(), want)


@pytest.mark.parametrize("dim,vdim", [(32, 1), (64, 30), (128, 256), (256, 200), (128, 64)])
@pytest.mark.parametrize("dtype,act", [("float32", True), ("bfloat16", False)])
@pytest.mark.parametrize("in_order", [False, True])
def test_retention_of_prompts_in_chunks(dim, vdim, dtype, act, in_order):
    """Sequences of one token, a chunk, a chunk and one, several; fresh ones and ones with a state; a token whose values
    are infinite is not felt before it."""
    o = ops()
    g = torch.Generator().manual_seed(dim + vdim)
    H, new, starts, rot = 2, [1, 64, 65, 200, 130], [0, 7, 0, 64, 0], dim // 2
    n, decay = sum(new), torch.tensor([0.97, 0.3])
    rows = torch.randn(n, 2 * H * (dim + vdim), generator=g).to(getattr(torch, dtype))
    last = n - 20  # in the last sequence's last chunk but one
    rows[last, 2 * H * dim:2 * H * dim + H * vdim] = math.inf if not act else 1.0
    freq = 100.0 ** (-torch.arange(rot // 2, dtype=torch.float32) / rot)
    state = torch.randn(9, H, dim, vdim, generator=g)
    slots = [3, 0, 8, 5, 1]
    for s, st in zip(slots, starts):
        if st == 0:
            state[s] = 0.0
    chunks, first = o.scan_segments(new, o.RETENTION_CHUNK)
    sizes = o.retention_scratch(len(chunks), H, dim, vdim)
    o_raw = torch.full((n, H * vdim), 5.0, device=DEV)
    out = torch.empty(n, H * vdim, dtype=rows.dtype, device=DEV)
    got_state = state.to(DEV)
    pos = [st + t for st, c in zip(starts, new) for t in range(c)]
    seq = [i for i, c in enumerate(new) for _ in range(c)]
    side_by_side = {} if in_order else dict(
        chunks=torch.from_numpy(chunks).to(DEV), seq_first_chunk=torch.from_numpy(first).to(DEV),
        packed=torch.full((sizes[0],), math.nan, device=DEV), chunk_state=torch.full((sizes[1],), math.nan, device=DEV))
    o.retention(rows.to(DEV), freq.to(DEV), decay.to(DEV), got_state, i32(pos), i32(seq), i32(slots),
                i32([sum(new[:i]) for i in range(len(new))]), i32(starts), i32(new), o_raw, out, H, dim, vdim, rot, 1e-5,
                activation=act, **side_by_side)
    x = rows.double()
    x = x * torch.sigmoid(x) if act else x
    q, k = (x[:, i * H * dim:(i + 1) * H * dim].reshape(n, H, dim).clone() for i in (0, 1))
    v = x[:, 2 * H * dim:2 * H * dim + H * vdim].reshape(n, H, vdim)
    ang = torch.tensor(pos, dtype=torch.float32)[:, None] * freq[None, :]
    c, s = torch.cos(ang.double())[:, None], torch.sin(ang.double())[:, None]
    half = rot // 2
    for y in (q, k):
        a, b = y[..., :half].clone(), y[..., half:rot].clone()
        y[..., :half], y[..., half:rot] = a * c - b * s, b * c + a * s
    k = k * dim ** -0.5
    want, row = torch.empty(n, H, vdim, dtype=torch.float64), 0
    for i, cnt in enumerate(new):
        S = state[slots[i]].double()
        for _ in range(cnt):
            S = decay.double()[:, None, None] * S + k[row][:, :, None] * v[row][:, None, :]
            want[row] = torch.einsum("hdv,hd->hv", S, q[row])
            row += 1
        if torch.isfinite(S).all():
            err = (got_state[slots[i]].cpu().double() - S).abs().max() / S.abs().max()
            assert err < 2e-6, (i, float(err))
    fine = n if act else last
    err = (o_raw.cpu().double()[:fine] - want.reshape(n, -1)[:fine]).abs().max() / want[:fine].abs().max()
    assert err < 2e-6, float(err)  # sums of at most 64 + dim products of order one and a rounding per chunk: a few ulps
    assert act or not torch.isfinite(o_raw[last]).any()


@pytest.mark.parametrize("wave", [1, 3, 4])
def test_retention_chunks_in_waves(wave, monkeypatch):
    """More chunks than the scratch holds: the same bits, whether a wave ends inside a sequence or with it."""
    o = ops()
    g = torch.Generator().manual_seed(wave)
    H, dim, vdim, new, starts = 2, 64, 40, [130, 64, 1, 300], [0, 5, 0, 64]
    n = sum(new)
    rows, decay = torch.randn(n, 2 * H * (dim + vdim), generator=g).to(DEV), torch.tensor([0.97, 0.5], device=DEV)
    begin, freq = torch.randn(4, H, dim, vdim, generator=g), torch.ones(1, device=DEV)
    for s, st in enumerate(starts):
        begin[s] *= st > 0
    chunks, first = (torch.from_numpy(t).to(DEV) for t in o.scan_segments(new, o.RETENTION_CHUNK))
    tables = [i32(x) for x in ([st + t for st, c in zip(starts, new) for t in range(c)],
                               [i for i, c in enumerate(new) for _ in range(c)], [0, 1, 2, 3],
                               [sum(new[:i]) for i in range(len(new))], starts, new)]
    got = []
    for scratch in (o.RETENTION_SCRATCH, 4 * wave * H * (64 * (3 * dim + vdim) + dim * vdim)):
        monkeypatch.setattr(o, "RETENTION_SCRATCH", scratch)
        assert o.retention_wave(len(chunks), H, dim, vdim) == (len(chunks) if not got else wave)
        sizes = o.retention_scratch(len(chunks), H, dim, vdim)
        state, o_raw = begin.to(DEV), torch.full((n, H * vdim), 5.0, device=DEV)
        o.retention(rows, freq, decay, state, *tables, o_raw, torch.empty(n, H * vdim, device=DEV), H, dim, vdim, 0, 1e-5,
                    chunks=chunks, seq_first_chunk=first, packed=torch.full((sizes[0],), math.nan, device=DEV),
                    chunk_state=torch.full((sizes[1],), math.nan, device=DEV))
        got.append((o_raw, state))
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])


@pytest.mark.parametrize("dim,vdim", [(64, 64), (64, 200), (128, 264), (128, 384)])
@pytest.mark.parametrize("dtype,act", [("float32", True), ("bfloat16", False)])
def test_retention_of_prompts_in_pairs_of_chunks(dim, vdim, dtype, act):
    """The sizes that go to the tensor cores: tiles of 128 columns half full, full, one CTA's two and more."""
    test_retention_of_prompts_in_chunks(dim, vdim, dtype, act, False)


@pytest.mark.parametrize("dim,vdim", [(128, 8), (128, 40), (128, 56)])
@pytest.mark.parametrize("dtype,act", [("float32", True), ("bfloat16", False)])
def test_retention_of_prompts_in_pairs_of_chunks_with_few_values(dim, vdim, dtype, act):
    """A tile of 128 columns of which most are not there."""
    test_retention_of_prompts_in_chunks(dim, vdim, dtype, act, False)


@pytest.mark.parametrize("vdim", [8, 40, 64])
def test_retention_of_long_prompts_in_pairs_of_chunks_with_small_heads(vdim):
    """Heads of 64 keys and few values go by pairs where sequences are long and many CTAs come of them: against the kernel
    that works the tokens in order."""
    o = ops()
    g = torch.Generator().manual_seed(vdim)
    H, dim, new, starts = 4, 64, [1500, 129], [0, 70]
    n = sum(new)
    chunks, first = (torch.from_numpy(t).to(DEV) for t in o.scan_segments(new, o.RETENTION_CHUNK))
    by_pairs, one_by_one = (o.retention_launches(c, s, H, dim, vdim, 20) for c, s in ((len(chunks), 2), (len(chunks), 9)))
    assert (by_pairs, one_by_one) == (4 * 2 + 1, 4 * 2 + 1) and o.retention_launches(len(chunks), 2, H, dim, vdim, 3) == 4 * 14 + 1
    rows = torch.randn(n, 2 * H * (dim + vdim), generator=g).to(DEV)
    decay, freq = torch.tensor([0.97, 0.5, 0.999, 0.9], device=DEV), torch.ones(1, device=DEV)
    begin = torch.randn(2, H, dim, vdim, generator=g)
    begin[0] = 0.0
    tables = [i32(x) for x in ([st + t for st, c in zip(starts, new) for t in range(c)], [0] * new[0] + [1] * new[1], [0, 1],
                               [0, new[0]], starts, new)]
    sizes = o.retention_scratch(len(chunks), H, dim, vdim)
    got = []
    for side in (dict(chunks=chunks, seq_first_chunk=first, packed=torch.full((sizes[0],), math.nan, device=DEV),
                      chunk_state=torch.full((sizes[1],), math.nan, device=DEV)), {}):
        state, o_raw = begin.to(DEV), torch.full((n, H * vdim), 5.0, device=DEV)
        o.retention(rows, freq, decay, state, *tables, o_raw, torch.empty(n, H * vdim, device=DEV), H, dim, vdim, 0, 1e-5, **side)
        got.append((o_raw, state))
    o.check_status(DEV)
    for x, y in zip(*got):  # (each within 2e-6 of 64 bits, as above)
        assert float((x - y).abs().max() / y.abs().max()) < 4e-6


@pytest.mark.parametrize("wave", [2, 3, 5])
def test_retention_pairs_of_chunks_in_waves(wave, monkeypatch):
    """The same bits however many pairs the scratch holds, with more sequences than a warp looks through at once."""
    o = ops()
    g = torch.Generator().manual_seed(wave)
    H, dim, vdim, new = 2, 64, 72, [130, 64, 1, 300] + [3, 70, 129] * 12
    starts = [0, 5, 0, 64] + [0, 9, 0] * 12
    n, seqs = sum(new), len(new)
    rows, decay = torch.randn(n, 2 * H * (dim + vdim), generator=g).to(DEV), torch.tensor([0.97, 0.5], device=DEV)
    begin, freq = torch.randn(seqs, H, dim, vdim, generator=g), torch.ones(1, device=DEV)
    for s, st in enumerate(starts):
        begin[s] *= st > 0
    chunks, first = (torch.from_numpy(t).to(DEV) for t in o.scan_segments(new, o.RETENTION_CHUNK))
    tables = [i32(x) for x in ([st + t for st, c in zip(starts, new) for t in range(c)],
                               [i for i, c in enumerate(new) for _ in range(c)], range(seqs),
                               [sum(new[:i]) for i in range(seqs)], starts, new)]
    got = []
    for scratch in (o.RETENTION_SCRATCH, 4 * wave * H * (64 * (3 * dim + vdim) + dim * vdim)):
        monkeypatch.setattr(o, "RETENTION_SCRATCH", scratch)
        sizes = o.retention_scratch(len(chunks), H, dim, vdim)
        state, o_raw = begin.to(DEV), torch.full((n, H * vdim), 5.0, device=DEV)
        o.retention(rows, freq, decay, state, *tables, o_raw, torch.empty(n, H * vdim, device=DEV), H, dim, vdim, 0, 1e-5,
                    chunks=chunks, seq_first_chunk=first, packed=torch.full((sizes[0],), math.nan, device=DEV),
                    chunk_state=torch.full((sizes[1],), math.nan, device=DEV))
        got.append((o_raw, state))
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1])
    assert got[0][0].isfinite().all() and got[0][1].isfinite().all()


@pytest.mark.parametrize("dim,vdim,taps", [(64, 30, 4), (128, 128, 4), (64, 200, 1), (128, 64, 3)])
@pytest.mark.parametrize("slow,alike", [(True, False), (False, False), (True, True)])
def test_delta_rule_of_prompts_in_chunks(dim, vdim, taps, slow, alike):
    """Against the walk token by token and the recurrence in 64 bits: sequences of one token, a chunk, a chunk and one,
    several, that go on from states and convolution inputs; decays near one, and fast ones among which some are zero; keys nearly
    alike with strong writes, which the triangle's inverse has to stand."""
    o = ops()
    g = torch.Generator().manual_seed(dim + vdim + taps)
    H, G, new = 4, 2, [1, 64, 65, 200, 130]
    n, channels = sum(new), 2 * G * dim + H * vdim
    rows = torch.randn(n, channels + H * vdim + 2 * H, generator=g)
    if not slow:
        rows[70:90, -1] = 1e4  # the last head's decay is zero there
    if alike:
        rows[:, G * dim:2 * G * dim] += 3.0 * torch.randn(1, G * dim, generator=g)
        rows[:, -2 * H:-H] += 4.0
    conv = torch.randn(channels, taps, generator=g).to(DEV)
    a_log = (torch.empty(H).uniform_(-7.0, -4.0, generator=g) if slow else torch.empty(H).uniform_(-1.0, 1.0, generator=g)).to(DEV)
    bias = torch.empty(H).uniform_(-1.0, 1.0, generator=g).to(DEV)
    begin = torch.randn(9, H, dim, vdim, generator=g) * 0.3
    tails = torch.randn(9, max(taps - 1, 1), channels, generator=g)
    slots, first, count = i32([3, 0, 8, 5, 1]), i32([sum(new[:i]) for i in range(len(new))]), i32(new)
    pos, seq = i32([t + 9 for c in new for t in range(c)]), i32([i for i, c in enumerate(new) for _ in range(c)])
    rd = rows.to(DEV)
    qkv, beta_g = torch.empty(n, channels, device=DEV), torch.empty(n, 2 * H, device=DEV)
    state, tail, walked = begin.to(DEV), tails.to(DEV), torch.empty(n, H * vdim, device=DEV)
    o.delta_prep(rd, conv, tail, a_log, bias, pos, seq, slots, first, count, qkv, beta_g, H, G, dim, vdim, 1e-6, dim ** -0.5)
    o.delta_scan(qkv, beta_g, state, pos, seq, slots, first, count, walked, H, G, dim, vdim)
    chunks, first_chunk = o.scan_segments(new, o.DELTA_CHUNK)
    state2, tail2, got = begin.to(DEV), tails.to(DEV), torch.full((n, H * vdim), math.nan, device=DEV)
    o.delta_prompt(rd, conv, tail2, a_log, bias, state2, pos, seq, slots, first, count, torch.from_numpy(chunks).to(DEV),
                   torch.from_numpy(first_chunk).to(DEV),
                   lambda name, shape, dtype: torch.full(shape, math.nan, dtype=dtype, device=DEV), got, H, G, dim, vdim,
                   1e-6, dim ** -0.5)
    assert torch.equal(tail, tail2)
    x, bg = qkv.double().cpu(), beta_g.double().cpu()
    q, k = (x[:, i * G * dim:(i + 1) * G * dim].view(n, G, dim).repeat_interleave(H // G, 1) for i in (0, 1))
    v, want, row = x[:, 2 * G * dim:].view(n, H, vdim), torch.empty(n, H, vdim, dtype=torch.float64), 0
    finals = begin.double().clone()
    for i, c in enumerate(new):
        S = begin[int(slots[i])].double()
        for _ in range(c):
            S = bg[row, H:, None, None] * S
            u = bg[row, :H, None] * (v[row] - torch.einsum("hdv,hd->hv", S, k[row]))
            S = S + k[row][:, :, None] * u[:, None, :]
            want[row] = torch.einsum("hdv,hd->hv", S, q[row])
            row += 1
        finals[int(slots[i])] = S
    if alike:
        assert (k[70:100, None] * k[None, 70:100]).sum(-1).mean() > 0.5
    # (a few hundred float32 roundings of values of order one, on either way: 1e-5 of the largest is some 80 ulps)
    for y, s in ((walked, state), (got, state2)):
        assert (y.cpu().double() - want.reshape(n, -1)).abs().max() < 1e-5 * want.abs().max()
        assert (s.cpu().double() - finals).abs().max() < 1e-5 * finals.abs().max()


@pytest.mark.parametrize("wave", [1, 3, 4])
def test_delta_rule_chunks_in_waves(wave, monkeypatch):
    """More chunks than the scratch holds: the same bits, whether a wave ends inside a sequence or with it."""
    o = ops()
    g = torch.Generator().manual_seed(wave)
    H, G, dim, vdim, taps, new = 2, 1, 64, 40, 4, [130, 64, 1, 300]
    n, channels = sum(new), 2 * G * dim + H * vdim
    rows = torch.randn(n, channels + H * vdim + 2 * H, generator=g).to(DEV)
    conv, a_log, bias = torch.randn(channels, taps, generator=g).to(DEV), torch.full((H,), -2.0, device=DEV), torch.zeros(H, device=DEV)
    begin, tails = torch.randn(4, H, dim, vdim, generator=g) * 0.3, torch.randn(4, taps - 1, channels, generator=g)
    chunks, first = (torch.from_numpy(t).to(DEV) for t in o.scan_segments(new, o.DELTA_CHUNK))
    tables = [i32(x) for x in ([t + 9 for c in new for t in range(c)], [i for i, c in enumerate(new) for _ in range(c)],
                               [0, 1, 2, 3], [sum(new[:i]) for i in range(len(new))], new)]
    got = []
    held = sum(math.prod(shape) * dtype.itemsize for _, shape, dtype in o.delta_scratch(wave, H, G, dim, vdim))
    for scratch in (o.DELTA_SCRATCH, held):
        monkeypatch.setattr(o, "DELTA_SCRATCH", scratch)
        asked = []

        def buffer(name, shape, dtype):
            asked.append(shape[0])
            return torch.full(shape, math.nan, dtype=dtype, device=DEV)

        state, tail, o_raw = begin.to(DEV), tails.to(DEV), torch.full((n, H * vdim), 5.0, device=DEV)
        o.delta_prompt(rows, conv, tail, a_log, bias, state, *tables, chunks, first, buffer, o_raw, H, G, dim, vdim, 1e-6, 1.0)
        assert asked == [wave if got else len(chunks)] * 6
        got.append((o_raw, state, tail))
    for one, other in zip(*got):
        assert torch.equal(one, other)


@pytest.mark.parametrize("column", [-1, -3])  # the last head's decay gate, and its strength of writing
def test_a_gate_of_the_delta_rule_that_is_no_number(column):
    """It is seen from its token on, as in the walk, and not before it."""
    o = ops()
    g = torch.Generator().manual_seed(7)
    H, G, dim, vdim, taps, n, at = 2, 1, 64, 32, 4, 200, 71
    channels = 2 * G * dim + H * vdim
    rows = torch.randn(n, channels + H * vdim + 2 * H, generator=g)
    rows[at, column] = math.nan
    conv, tails = torch.randn(channels, taps, generator=g).to(DEV), torch.zeros(1, taps - 1, channels, device=DEV)
    a_log, bias, rd = torch.full((H,), -2.0, device=DEV), torch.zeros(H, device=DEV), rows.to(DEV)
    slots, first, count, pos, seq = i32([0]), i32([0]), i32([n]), i32(list(range(n))), i32([0] * n)
    qkv, beta_g = torch.empty(n, channels, device=DEV), torch.empty(n, 2 * H, device=DEV)
    state, walked = torch.zeros(1, H, dim, vdim, device=DEV), torch.empty(n, H * vdim, device=DEV)
    o.delta_prep(rd, conv, tails.clone(), a_log, bias, pos, seq, slots, first, count, qkv, beta_g, H, G, dim, vdim, 1e-6, 1.0)
    o.delta_scan(qkv, beta_g, state, pos, seq, slots, first, count, walked, H, G, dim, vdim)
    chunks, first_chunk = o.scan_segments([n], o.DELTA_CHUNK)
    state2, got = torch.zeros(1, H, dim, vdim, device=DEV), torch.full((n, H * vdim), 7.0, device=DEV)
    o.delta_prompt(rd, conv, tails.clone(), a_log, bias, state2, pos, seq, slots, first, count,
                   torch.from_numpy(chunks).to(DEV), torch.from_numpy(first_chunk).to(DEV),
                   lambda name, shape, dtype: torch.full(shape, math.nan, dtype=dtype, device=DEV), got, H, G, dim, vdim,
                   1e-6, 1.0)
    bad = torch.zeros(n, H, vdim, dtype=torch.bool)
    bad[at:, -1] = True
    for y, s in ((walked, state), (got, state2)):
        assert torch.equal(torch.isnan(y.cpu()).view(n, H, vdim), bad)
        assert torch.equal(torch.isnan(s.cpu())[0].flatten(1).all(1), bad[-1, :, 0]) and not torch.isnan(s[0, ~bad[-1, :, 0]]).any()
    assert (walked - got)[~bad.view(n, -1)].abs().max() < 1e-5 * walked[~bad.view(n, -1)].abs().max()


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("width,groups", [(4, 1), (1028, 1), (2048, 4), (4096, 1), (8192, 2), (8196, 3), (516, 129), (30, 5)])
@pytest.mark.parametrize("n", [1, 70])
def test_norms_and_gather_of_rows(dtype, width, groups, n):
    """Rows that are held whole in registers, in one, two, four and eight pieces, and rows that are not."""
    o, dt = ops(), getattr(torch, dtype)
    g = torch.Generator().manual_seed(width + n)
    x, w = torch.randn(n + 3, width, generator=g), torch.randn(width, generator=g)
    rows = torch.randperm(n + 3, generator=g)[:n].to(torch.int32)
    pick = x[rows.long()].double()
    out = torch.empty(n, width, dtype=dt, device=DEV)
    o.rmsnorm(x.to(DEV), w.to(DEV), 1e-5, out, rows.to(DEV))
    close(out, pick / torch.sqrt((pick * pick).mean(-1, keepdim=True) + 1e-5) * w.double(), dtype, "norm")
    o.group_rmsnorm(x.to(DEV), w.to(DEV), 1e-5, groups, out, rows.to(DEV))
    y = pick.view(n, groups, -1)
    close(out, (y / torch.sqrt((y * y).mean(-1, keepdim=True) + 1e-5)).view(n, width) * w.double(), dtype, "groups")
    table, hidden = x.to(dt), torch.empty(n, width, device=DEV)
    status = torch.zeros(1, dtype=torch.int32, device=DEV)
    o.embed(table.to(DEV), rows.to(DEV), hidden, status)
    assert torch.equal(hidden.cpu(), table[rows.long()].float()) and int(status) == 0


@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
@pytest.mark.parametrize("H,vdim", [(2, 4), (4, 128), (2, 132), (2, 256), (2, 512), (2, 516), (3, 30)])
def test_heads_normed_and_gated(dtype, H, vdim):
    o, dt = ops(), getattr(torch, dtype)
    g = torch.Generator().manual_seed(H * vdim)
    n, off = 9, 8
    raw, rows = torch.randn(n, H * vdim, generator=g), torch.randn(n, off + H * vdim + 4, generator=g)
    pos = i32([0, 1, -1, 3, 4, 5, 6, 7, 8])
    z, y = rows[:, off:off + H * vdim].double().view(n, H, vdim), raw.double().view(n, H, vdim)
    y = y / torch.sqrt((y * y).mean(-1, keepdim=True) + 1e-5)
    live = (pos.cpu() >= 0).double()[:, None]
    for w, finish, f in ((torch.randn(vdim, generator=g), o.delta_finish, z * torch.sigmoid(z)),
                         (torch.randn(H * vdim, generator=g), o.memory_finish, torch.sigmoid(z))):
        out = torch.full((n, H * vdim), 5.0, dtype=dt, device=DEV)
        args = (raw.to(DEV), rows.to(DEV), off, w.to(DEV), pos, out, H, vdim, 1e-5)
        finish(*args)
        close(out, (y * w.double().view(-1, vdim) * f).view(n, -1) * live, dtype, finish.__name__)


# 14 tiles of rows by 8 of 256 columns (an SM for each CTA); 19 by 10 (two on an SM, the last pair's second CTA without
# rows); rows of the output off 16-byte boundaries; tails of K
@pytest.mark.parametrize("m,n,k", [(1700, 1928, 2056), (2400, 2312, 520), (2300, 2306, 584), (2560, 4096, 1024)])
def test_products_on_pairs_of_ctas(m, n, k):
    """Storing, adding and gated products large enough for pairs of CTAs against 64 bits.  A float32 sum of k products,
    however it is grouped, is within k 2^-23 of the sum of their sizes (2^-23: sums that are cut, not rounded)."""
    o = ops()
    g = torch.Generator(device=DEV).manual_seed(m + n + k)
    a = torch.randn(m, k, generator=g, device=DEV).bfloat16()
    w = (torch.randn(n, k, generator=g, device=DEV) / math.sqrt(k)).bfloat16()
    bias = torch.randn(n, generator=g, device=DEV)
    want = a.double() @ w.double().t() + bias.double()
    bound = k * 2.0 ** -23 * (a.double().abs() @ w.double().abs().t() + bias.double().abs()) + 1e-12
    out = torch.full((m, n), 7.0, device=DEV)
    o.gemm_tc(a, w, bias, out, o.STORE_F32)
    assert bool(((out.double() - want).abs() <= bound).all())
    base = torch.randn(m, n, generator=g, device=DEV)
    acc = base.clone()
    o.gemm_tc(a, w, bias, acc, o.ADD_F32)
    total = base.double() + want
    assert bool(((acc.double() - total).abs() <= bound + 2.0 ** -23 * total.abs()).all())
    half = torch.full((m, n), 7.0, dtype=torch.bfloat16, device=DEV)
    o.gemm_tc(a, w, bias, half, o.STORE)
    assert bool(((half.double() - want).abs() <= bound + 2.0 ** -8 * want.abs()).all())
    gated = torch.full((m, n // 2), 7.0, dtype=torch.bfloat16, device=DEV)
    o.gemm_tc(a, w, bias, gated, o.GEMM_GATED)
    close(gated, P.swiglu(want[:, :n // 2], want[:, n // 2:]), "bfloat16", "gated product of pairs")
    o.check_status(DEV)


@pytest.mark.parametrize("nq,nkv,d,m,k", [(16, 4, 128, 1100, 2048), (35, 3, 64, 2500, 576)])
def test_qkv_products_on_pairs_of_ctas(nq, nkv, d, m, k):
    """Heads rotated and stored from tiles of 256 columns: the same bits as the tiles of 128 that fewer rows take."""
    o = ops()
    g = torch.Generator(device=DEV).manual_seed(nq + m)
    n, page = (nq + 2 * nkv) * d, 64
    w = (torch.randn(n, k, generator=g, device=DEV) / math.sqrt(k)).bfloat16()
    bias = torch.randn(n, generator=g, device=DEV)
    x = torch.randn(m, k, generator=g, device=DEV).bfloat16()
    cos, sin = (t.float().to(DEV) for t in P.rope_tables(m, d, 10000.0))
    pos = torch.arange(m, dtype=torch.int32, device=DEV)
    pos[m - 1] = -1  # a padding row
    pages = -(-m // page)
    table = torch.randperm(pages, generator=g, device=DEV).int().view(1, -1)

    def product(rows):
        q = torch.full((m, nq * d), 9.0, dtype=torch.bfloat16, device=DEV)
        kc, vc = (torch.zeros(pages, nkv, page, d, dtype=torch.bfloat16, device=DEV) for _ in range(2))
        for r in range(0, m, rows):
            e = min(r + rows, m)
            o.gemm_tc(x[r:e], w, bias, q[r:e], o.GEMM_QKV, token_pos=pos[r:e], token_seq=torch.zeros_like(pos[r:e]),
                      page_table=table, cos=cos, sin=sin, k_cache=kc, v_cache=vc, heads=nq, kv_heads=nkv, head_dim=d,
                      page_size=page)
        return q, kc, vc

    for whole, parts in zip(product(m), product(128)):
        assert torch.equal(whole, parts)
    o.check_status(DEV)


@pytest.mark.parametrize("dim,vdim", [(64, 4), (64, 136), (128, 72), (128, 300)])
def test_delta_rule_chunks_at_the_edges_of_their_tiles(dim, vdim):
    """Columns that end inside an octet, a CTA's 64 and a tile of 128, chunks that end at their first and last token, a head
    per key head: against the recurrence in 64 bits.  A value that is no number is felt by its own column from its token on."""
    o = ops()
    g = torch.Generator().manual_seed(dim + vdim)
    H, G, taps, new, at = 2, 2, 1, [65, 1, 63, 128, 129], 100 + 129
    n, channels = sum(new), 2 * G * dim + H * vdim
    rows = torch.randn(n, channels + H * vdim + 2 * H, generator=g)
    conv, a_log, bias = torch.ones(channels, taps, device=DEV), torch.tensor([-5.0, 0.5], device=DEV), torch.zeros(H, device=DEV)
    begin, tails = torch.randn(len(new), H, dim, vdim, generator=g) * 0.3, torch.zeros(len(new), 1, channels, device=DEV)
    first = [sum(new[:i]) for i in range(len(new))]
    pos, seq = i32([t for c in new for t in range(c)]), i32([i for i, c in enumerate(new) for _ in range(c)])
    chunks, first_chunk = (torch.from_numpy(t).to(DEV) for t in o.scan_segments(new, o.DELTA_CHUNK))

    def run(x):
        state, out = begin.to(DEV), torch.full((n, H * vdim), math.nan, device=DEV)
        o.delta_prompt(x.to(DEV), conv, tails, a_log, bias, state, pos, seq, i32(range(len(new))), i32(first), i32(new), chunks,
                       first_chunk, lambda name, shape, dtype: torch.full(shape, math.nan, dtype=dtype, device=DEV), out, H, G,
                       dim, vdim, 1e-6, dim ** -0.5)
        return out.view(n, H, vdim).cpu(), state.cpu()

    out, state = run(rows)
    x = torch.nn.functional.silu(rows[:, :channels].double())
    q, k = (y / (y.pow(2).sum(-1, keepdim=True) + 1e-6).sqrt() for y in (x[:, :G * dim].view(n, G, dim), x[:, G * dim:2 * G * dim].view(n, G, dim)))
    v, beta = x[:, 2 * G * dim:].view(n, H, vdim), torch.sigmoid(rows[:, -2 * H:-H].double())
    decay = torch.exp(-torch.exp(a_log.cpu().double()) * torch.nn.functional.softplus(rows[:, -H:].double()))
    want, finals = torch.empty(n, H, vdim, dtype=torch.float64), []
    for i, c in enumerate(new):
        S = begin[i].double()
        for r in range(first[i], first[i] + c):
            S = decay[r, :, None, None] * S
            S = S + k[r][:, :, None] * (beta[r, :, None] * (v[r] - torch.einsum("hdv,hd->hv", S, k[r])))[:, None, :]
            want[r] = torch.einsum("hdv,hd->hv", S, q[r]) * dim ** -0.5
        finals.append(S)
    finals = torch.stack(finals)
    # (as test_delta_rule_of_prompts_in_chunks, and the float32 gates: a hundred roundings of logs of up to 5 a token, 1e-5 more)
    assert (out.double() - want).abs().max() < 2e-5 * want.abs().max()
    assert (state.double() - finals).abs().max() < 2e-5 * finals.abs().max()
    rows[at, 2 * G * dim + vdim + 3] = math.nan  # the last prompt but one, its token 100; head 1, column 3
    bad, bad_state = run(rows)
    hit = torch.zeros(n, H, vdim, dtype=torch.bool)
    hit[at:first[4], 1, 3] = True
    # (the column's earlier tokens of that chunk are summed in another order)
    assert torch.equal(torch.isnan(bad), hit) and (bad - out)[~hit].abs().max() < 1e-5 * out.abs().max()
    hit = torch.zeros_like(state, dtype=torch.bool)
    hit[3, 1, :, 3] = True
    assert torch.equal(torch.isnan(bad_state), hit) and torch.equal(bad_state[~hit], state[~hit])


def test_a_chunks_decays_are_rounded_once():
    """e^(c_last - c_j) of every chunk, as the solve leaves it for the walk, against 64-bit sums of the same logs: the difference is rounded
    to float32 once (half a unit in its last place) and the exponential is two units off at most."""
    o = ops()
    g = torch.Generator().manual_seed(3)
    H, G, dim, vdim, taps, n = 16, 1, 64, 32, 1, 512
    channels = 2 * G * dim + H * vdim
    rows = torch.randn(n, channels + H * vdim + 2 * H, generator=g).to(DEV)
    conv, tails = torch.ones(channels, taps, device=DEV), torch.zeros(1, 1, channels, device=DEV)
    a_log, bias = torch.linspace(-4.0, 0.5, H).to(DEV), torch.zeros(H, device=DEV)
    tables = [i32(x) for x in (range(n), [0] * n, [0], [0], [n])]
    qkv, beta_g = torch.empty(n, channels, device=DEV), torch.empty(n, 2 * H, device=DEV)
    o.delta_prep(rows, conv, tails.clone(), a_log, bias, *tables, qkv, beta_g, H, G, dim, vdim, 1e-6, 1.0)
    chunks, first = (torch.from_numpy(t).to(DEV) for t in o.scan_segments([n], o.DELTA_CHUNK))
    held = {}

    def buffer(name, shape, dtype):
        held[name] = torch.full(shape, math.nan, dtype=dtype, device=DEV)
        return held[name]

    o.delta_prompt(rows, conv, tails, a_log, bias, torch.zeros(1, H, dim, vdim, device=DEV), *tables, chunks, first, buffer,
                   torch.empty(n, H * vdim, device=DEV), H, G, dim, vdim, 1e-6, 1.0)
    got = held["delta_chunk_logs"].cpu().view(torch.float32).view(n // 64, H, 128)[..., :64].double()
    c = torch.log(beta_g[:, H:].cpu().double()).view(n // 64, 64, H).cumsum(1).transpose(1, 2)
    d = c[..., -1:] - c
    half_unit = torch.exp2(torch.floor(torch.log2(d.abs().clamp(min=2.0**-126))) - 24)
    assert (d < -32).sum() > 500 and ((got / d.exp() - 1).abs() <= 1.01 * half_unit + 2.0**-22)[d > -80].all()
