"""Kernels of decode steps (and the router and the merge that prompts share with them) at the sizes where they can go wrong."""
import math

import pytest
import torch

from test_kernels_gpu import DEV, ops

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 9, 300, 511, 512, 517])
@pytest.mark.parametrize("width,experts,top", [(40, 11, 4), (36, 3, 3), (30, 65, 2), (516, 33, 33)])
@pytest.mark.parametrize("sigmoid", [False, True])
def test_router_of_few_and_of_many_tokens(n, width, experts, top, sigmoid):
    """One token a CTA and eight: the last CTA's missing tokens, experts that fill no round of the warps, ties, rows off
    the 16-byte boundary, padding rows, a token whose logits are no numbers."""
    o = ops()
    g = torch.Generator().manual_seed(n + width)
    h, wr, br = torch.randn(n, width, generator=g), torch.randn(experts, width, generator=g), torch.randn(experts, generator=g)
    wr[experts - 1], br[experts - 1] = wr[0], br[0]  # a tie
    pos = torch.zeros(n, dtype=torch.int32)
    if n > 8:
        pos[5], pos[n - 1] = -1, -1
        h[6] = math.nan
    ids = torch.full((n, top), 77, dtype=torch.int32, device=DEV)
    weights = torch.full((n, top), 7.0, device=DEV)
    o.moe_route(h.to(DEV), wr.to(DEV), br.to(DEV), pos.to(DEV), ids, weights, top, sigmoid_scores=sigmoid)
    ids, weights = ids.cpu(), weights.cpu().double()
    z = h.double() @ wr.double().t() + br.double()
    for t in range(n):
        if pos[t] < 0:
            assert ids[t].tolist() == [0] * top and weights[t].tolist() == [0.0] * top
        elif h[t].isnan().any():
            assert weights[t].isnan().all() and all(0 <= i < experts for i in ids[t].tolist())
        else:
            # (float32 sums of `width` products: 1e-4 of logits of about sqrt(width))
            got = z[t, ids[t].long()]
            want = torch.sort(z[t], descending=True).values[:top]
            assert len(set(ids[t].tolist())) == top and torch.allclose(got, want, atol=1e-4 * math.sqrt(width))
            if 0 in ids[t].tolist() and experts - 1 in ids[t].tolist():
                assert ids[t].tolist().index(0) < ids[t].tolist().index(experts - 1)
            share = torch.sigmoid(got) if sigmoid else torch.softmax(got, 0)
            assert torch.allclose(weights[t], share, atol=1e-4)


@pytest.mark.parametrize("n", [3, 520])
@pytest.mark.parametrize("hidden", [-math.inf, torch.finfo(torch.float32).min])
@pytest.mark.parametrize("sigmoid", [False, True])
def test_router_with_experts_that_are_masked_out(n, hidden, sigmoid):
    """A bias of minus infinity, or of the type's lowest value, is a logit like any other: chosen last, by index, with no
    weight; a token with fewer other logits than choices still has numbers."""
    o = ops()
    g = torch.Generator().manual_seed(n)
    width, experts, top = 36, 40, 6
    h, wr, br = torch.randn(n, width, generator=g), torch.randn(experts, width, generator=g), torch.full((experts,), hidden)
    seen = [3, 17, 33, 38]
    br[seen] = torch.randn(4, generator=g)
    ids = torch.full((n, top), 77, dtype=torch.int32, device=DEV)
    weights = torch.full((n, top), 7.0, device=DEV)
    o.moe_route(h.to(DEV), wr.to(DEV), br.to(DEV), torch.zeros(n, dtype=torch.int32, device=DEV), ids, weights, top,
                sigmoid_scores=sigmoid)
    z = h.double() @ wr.double().t() + br.double()
    order = torch.sort(z[:, seen], descending=True).indices
    want = torch.tensor(seen)[order]
    assert torch.equal(ids[:, :4].cpu().long(), want) and (ids[:, 4:].cpu() == torch.tensor([0, 1])).all()
    got = z.gather(1, want)
    share = torch.sigmoid(got) if sigmoid else torch.softmax(got, 1)
    # (float32 sums of `width` products: 1e-4 of logits of about sqrt(width))
    assert torch.allclose(weights[:, :4].cpu().double(), share, atol=1e-4) and (weights[:, 4:] == 0.0).all()


@pytest.mark.parametrize("dim,rot,heads", [(16, 4, 3), (48, 16, 2), (144, 8, 5), (504, 8, 2)])
@pytest.mark.parametrize("splits", [2, 8, 9, 64])
@pytest.mark.parametrize("dtype", ["float32", "bfloat16"])
def test_merge_of_slices(dim, rot, heads, splits, dtype):
    """Attention in slices against the same in one: rows of one warp and of a CTA, slices that hold no key, rows that are
    no multiple of four."""
    o = ops()
    dt = getattr(torch, dtype)
    g = torch.Generator().manual_seed(dim + splits)
    lengths = [1, 64, 65, 300]
    n, row = len(lengths), dim + rot
    cache = torch.randn(16, 1, 64, row, generator=g).to(dt).to(DEV)
    table = torch.full((n, 5), -1, dtype=torch.int32)
    table.view(-1)[[0, 5, 10, 11, 15, 16, 17, 18, 19]] = torch.arange(9, dtype=torch.int32) + 2
    q = torch.randn(n, heads * row, generator=g).to(dt).to(DEV)
    pos = torch.tensor([length - 1 for length in lengths], dtype=torch.int32, device=DEV)
    seq, table = torch.arange(n, dtype=torch.int32, device=DEV), table.to(DEV)
    whole, cut = (torch.full((n, heads * dim), 9.0, dtype=dt, device=DEV) for _ in range(2))
    o.attention_latent(q, cache, pos, seq, table, whole, heads, dim, 0.2, 1, None)
    partial = torch.full((n * heads * splits * (dim + 2),), math.nan, device=DEV)
    o.attention_latent(q, cache, pos, seq, table, cut, heads, dim, 0.2, splits, partial)
    # float32: sums in another order; bfloat16: one rounding of the output
    assert torch.allclose(whole.float(), cut.float(), atol=2e-6 if dtype == "float32" else 2e-2)
    if dtype == "float32":
        for t, length in enumerate(lengths):
            rows = torch.cat([cache[int(p), 0] for p in table[t].cpu() if p >= 0])[:length].double()
            for h in range(heads):
                s = torch.softmax(rows @ q[t, h * row:(h + 1) * row].double() * 0.2, 0)
                assert torch.allclose(cut[t, h * dim:(h + 1) * dim].double(), s @ rows[:, :dim], atol=1e-5)


@pytest.mark.parametrize("dim", [66, 96, 128])
@pytest.mark.parametrize("splits", [3, 16])
def test_merge_of_many_rows_has_the_bits_of_few(dim, splits):
    """Rows of 65 to 128 values take a CTA each, or a warp each where they are many."""
    o = ops()
    g = torch.Generator().manual_seed(dim)
    n, heads, row = 270, 8, dim + 8
    cache = torch.randn(n, 1, 64, row, generator=g).to(DEV)
    q = torch.randn(n, heads * row, generator=g).to(DEV)
    pos = torch.randint(0, 64, (n,), generator=g).to(torch.int32).to(DEV)
    seq, table = torch.arange(n, dtype=torch.int32, device=DEV), torch.randperm(n, generator=g).to(torch.int32).view(n, 1).to(DEV)

    def run(a, b):
        out = torch.full((b - a, heads * dim), 9.0, device=DEV)
        partial = torch.full(((b - a) * heads * splits * (dim + 2),), math.nan, device=DEV)
        o.attention_latent(q[a:b], cache, pos[a:b], seq[:b - a], table[a:b], out, heads, dim, 0.2, splits, partial)
        return out
    assert torch.equal(run(0, n), torch.cat([run(0, 100), run(100, 249), run(249, n)]))


@pytest.mark.parametrize("m,n,k", [(1, 2048, 5632), (16, 520, 12288), (8, 2048, 5632), (20, 960, 2560), (33, 1024, 3200),
                                   (64, 2048, 8192), (5, 40, 12288)])
@pytest.mark.parametrize("emits", [False, True])
def test_adding_projection_whose_ctas_share_a_long_k(m, n, k, emits):
    """One launch in place of one per slice: parts of unequal length, units that fill no CTA, several tiles of rows, the
    next norm's values, and the same bits every time."""
    o = ops()
    g = torch.Generator().manual_seed(m + n + k)
    x = torch.randn(m, k, generator=g).bfloat16().to(DEV)
    w = (torch.randn(n, k, generator=g) / math.sqrt(k)).bfloat16().to(DEV)
    bias, old = torch.randn(n, generator=g).to(DEV), torch.randn(m, n, generator=g).to(DEV)
    floats, tiles = o.gemv_split_scratch(m, n, k, DEV)
    assert floats and tiles and o.gemv_slices(m, n, k, DEV) > 1
    split = (torch.full((floats,), math.nan, device=DEV), torch.zeros(tiles, dtype=torch.int32, device=DEV))
    want = old.double() + bias.double() + x.double() @ w.double().T
    emit_w = torch.rand(n, generator=g).to(DEV) + 0.5
    first = None
    for _ in range(3):
        emit = (torch.empty(m, n, dtype=torch.bfloat16, device=DEV), emit_w, torch.empty(m, n // 8, device=DEV)) if emits else None
        out = old.clone()
        o.gemv_bf16(w, bias, out, o.EPI_ADD_F32, x=x, emit=emit, split=split)
        first = out if first is None else first
        assert torch.equal(out, first) and int(split[1].abs().sum()) == 0
    # (float32 sums of products of bfloat16 values, cut off at 2^-23 of a running sum by the tensor cores: 96 of them a chain)
    assert float((out.double() - want).norm() / want.norm()) < 1e-6
    if emits:
        assert torch.equal(emit[0], (out * emit_w).bfloat16())
        assert torch.allclose(emit[2].double(), out.double().view(m, n // 8, 8).square().sum(-1), rtol=1e-6)
    cut = old.clone()
    o.gemv_bf16(w, bias, cut, o.EPI_ADD_F32, x=x)  # without the buffers: slices, as before
    assert torch.allclose(cut, out, atol=1e-5)
    small = (split[0][:floats - 1], split[1])  # buffers too small for it: slices
    again = old.clone()
    o.gemv_bf16(w, bias, again, o.EPI_ADD_F32, x=x, split=small)
    assert torch.equal(again, cut)
    o.check_status(DEV)


@pytest.mark.parametrize("m", [1, 8, 9, 16])
@pytest.mark.parametrize("n,k", [(2368, 2048), (2376, 2048), (6144, 1552), (2400, 3072), (9600, 2064)])
def test_projection_of_many_output_features(m, n, k):
    """A unit at a time, K shared by the warps: shares of K of unequal length, units that fill no round of the CTAs, each
    epilogue."""
    o = ops()
    g = torch.Generator().manual_seed(m + n + k)
    x = torch.randn(m, k, generator=g).bfloat16().to(DEV)
    w = (torch.randn(n, k, generator=g) / math.sqrt(k)).bfloat16().to(DEV)
    bias = torch.randn(n, generator=g).to(DEV)
    assert o.gemv_kind(m, n, k, o.EPI_STORE, DEV) == 1
    z = x.double() @ w.double().T + bias.double()
    out = torch.full((m, n), math.nan, device=DEV)
    o.gemv_bf16(w, bias, out, o.EPI_STORE_F32, x=x)
    assert float((out.double() - z).norm() / z.norm()) < 1e-6  # (float32 sums; their chains are 24 products of 16 values)
    half = torch.full((m, n), math.nan, dtype=torch.bfloat16, device=DEV)
    o.gemv_bf16(w, bias, half, o.EPI_STORE, x=x)
    assert torch.equal(half, out.bfloat16())
    o.gemv_bf16(w, bias, half, o.EPI_STORE, x=x, act=o.GEMM_ACT_RELU2)
    assert torch.equal(half, torch.relu(out).square().bfloat16())
    gated = torch.full((m, n // 2), math.nan, dtype=torch.bfloat16, device=DEV)
    o.gemv_bf16(w, bias, gated, o.EPI_GATED, x=x)
    want = torch.nn.functional.silu(z[:, :n // 2]) * z[:, n // 2:]
    assert torch.allclose(gated.double(), want, rtol=2.0 ** -8, atol=1e-5)  # (one rounding to bfloat16)
    old = torch.empty_like(out)
    o.gemv_bf16(w, bias, old, o.EPI_STORE_F32, x=x, rows_kernel=False)
    assert torch.allclose(old, out, atol=2e-5)
    o.check_status(DEV)


@pytest.mark.parametrize("heads", [1, 8, 16, 17, 32])
@pytest.mark.parametrize("dk,dv", [(576, 512), (288, 256), (24, 16), (72, 64), (56, 48)])
@pytest.mark.parametrize("window", [0, 1, 70])
def test_latent_attention_of_single_tokens(heads, dk, dv, window):
    """Against 64 bits: pages that are not full, a slot of a page that no token has filled or that the window hides (NaN
    there), more pages than the ring holds, slices without a key, padding rows, gates and sinks."""
    o = ops()
    assert o.attention_latent_decode_takes(heads, dk, dv, 64) and not o.attention_latent_decode_takes(33, dk, dv, 64)
    g = torch.Generator().manual_seed(heads + dk + window)
    lengths = [1, 64, 65, 0, 130, 700]
    n, cols = len(lengths), 11
    cache = torch.full((40, 1, 64, dk), math.nan, dtype=torch.bfloat16)
    table = torch.full((n, cols), -1, dtype=torch.int32)
    kept, page = [], 3
    for t, length in enumerate(lengths):
        rows = torch.randn(length, dk, generator=g).bfloat16()
        kept.append(rows.double())
        for p in range(-(-length // 64)):
            table[t, p] = page
            part = rows[p * 64:(p + 1) * 64]
            cache[page, 0, :len(part)] = part
            page += 1
        if window:  # (rows that the token does not see any more)
            for i in range(0, max(0, length - window)):
                cache[int(table[t, i // 64]), 0, i % 64] = math.nan
    q = torch.randn(n, heads * dk, generator=g).bfloat16()
    gate, sink = torch.rand(n, heads, generator=g), torch.randn(heads, generator=g)
    pos = torch.tensor([length - 1 for length in lengths], dtype=torch.int32)
    d = lambda t: t.to(DEV)
    scale = dk ** -0.5
    for splits in (1, 2, 7, 64):
        for with_gate, with_sink in ((False, False), (True, True)):
            out = torch.full((n, heads * dv), 9.0, dtype=torch.bfloat16, device=DEV)
            partial = torch.full((n * heads * splits * (dv + 2),), math.nan, device=DEV) if splits > 1 else None
            o.attention_latent_decode(d(q), d(cache), d(pos), torch.arange(n, dtype=torch.int32, device=DEV), d(table), out,
                                      heads, dv, scale, splits, partial, window, d(gate) if with_gate else None,
                                      d(sink) if with_sink else None)
            got = out.cpu().double().view(n, heads, dv)
            for t, length in enumerate(lengths):
                if not length:
                    continue
                rows = kept[t][max(0, length - window) if window else 0:]
                s = q[t].double().view(heads, dk) @ rows.T * scale
                if with_sink:
                    s = torch.cat([s, sink.double()[:, None]], 1)
                p = torch.softmax(s, 1)[:, :rows.shape[0]]
                want = p @ rows[:, :dv] * (gate[t].double()[:, None] if with_gate else 1.0)
                # (weights and outputs rounded to bfloat16, half a unit in eight bits each: 2^-7 of sums of |p v| together)
                bound = 2.0 ** -7 * (p @ rows[:, :dv].abs()) * (gate[t].double()[:, None] if with_gate else 1.0) + 1e-4
                assert ((got[t] - want).abs() <= bound).all(), (t, splits)
    o.check_status(DEV)


@pytest.mark.parametrize("heads,dk,dv", [(16, 576, 512), (8, 288, 256), (17, 72, 64)])
@pytest.mark.parametrize("window", [130, 330, 450])
def test_latent_attention_of_single_tokens_under_windows_of_more_pages_than_the_ring(heads, dk, dv, window):
    """The first page of a window has hidden rows, is zeroed there, and its place is filled again: against 64 bits, and the same
    bits whatever the hidden rows hold."""
    o = ops()
    g = torch.Generator().manual_seed(heads + window)
    lengths, cols = [700, 461, 512, 640, 333], 11
    n = len(lengths)
    rows = torch.randn(n, cols * 64, dk, generator=g).bfloat16()
    table = torch.randperm(n * cols, generator=g).to(torch.int32).view(n, cols)
    q = torch.randn(n, heads * dk, generator=g).bfloat16()
    scale = dk ** -0.5
    d = lambda t: t.to(DEV)
    for splits in (1, 2):
        first = None
        for hidden in (0.0, 1e4, math.nan):
            cache = torch.full((n * cols, 1, 64, dk), hidden, dtype=torch.bfloat16)
            for t, length in enumerate(lengths):
                for i in range(length - window if length > window else 0, length):
                    cache[int(table[t, i // 64]), 0, i % 64] = rows[t, i]
            out = torch.full((n, heads * dv), 9.0, dtype=torch.bfloat16, device=DEV)
            partial = torch.full((n * heads * splits * (dv + 2),), math.nan, device=DEV) if splits > 1 else None
            o.attention_latent_decode(d(q), d(cache), d(torch.tensor(lengths, dtype=torch.int32) - 1),
                                      torch.arange(n, dtype=torch.int32, device=DEV), d(table), out, heads, dv, scale, splits,
                                      partial, window)
            first = out.clone() if first is None else first
            assert torch.equal(out, first), (splits, hidden)
        for t, length in enumerate(lengths):
            seen = rows[t, max(0, length - window):length].double()
            p = torch.softmax(q[t].double().view(heads, dk) @ seen.T * scale, 1)
            # (weights and outputs rounded to bfloat16, half a unit in eight bits each: 2^-7 of sums of |p v| together)
            bound = 2.0 ** -7 * (p @ seen[:, :dv].abs()) + 1e-4
            assert ((first[t].cpu().double().view(heads, dv) - p @ seen[:, :dv]).abs() <= bound).all(), (t, splits)
    o.check_status(DEV)


@pytest.mark.parametrize("m", [1, 7, 8, 9, 16])
@pytest.mark.parametrize("heads,n,k", [(3, 8, 32), (2, 40, 96), (5, 24, 160), (16, 512, 128), (4, 128, 512), (2, 16, 544), (3, 12, 64)])
@pytest.mark.parametrize("gate", [False, True])
def test_small_matrix_per_head_on_few_rows(m, heads, n, k, gate):
    """Pieces of K that fill no round, columns that fill no CTA, sizes and strides that are left to the CUDA cores, rows
    and outputs with values of others between them."""
    o = ops()
    g = torch.Generator().manual_seed(m + n + k)
    for a_head, out_head in ((k, n), (k + 8, n + 8), (k + 4, n + 1)):
        a = torch.randn(m, heads * a_head, generator=g).bfloat16()
        w = (torch.randn(heads, n, k, generator=g) / math.sqrt(k)).bfloat16()
        logits = torch.randn(m, heads * n + 3, generator=g) if gate else None
        out = torch.full((m, heads * out_head), 7.0, dtype=torch.bfloat16, device=DEV)
        o.batched_linear(a.to(DEV), a_head, w.to(DEV), out, out_head, gate=logits.to(DEV) if gate else None, gate_off=3 if gate else 0)
        want = torch.einsum("mhk,hnk->mhn", a.view(m, heads, a_head)[..., :k].double(), w.double())
        if gate:
            want = want * torch.sigmoid(logits[:, 3:].double()).view(m, heads, n)
        got = out.cpu().double().view(m, heads, out_head)
        assert torch.allclose(got[..., :n], want, rtol=2.0 ** -8, atol=1e-5)  # (one rounding to bfloat16)
        assert (got[..., n:] == 7.0).all()


@pytest.mark.parametrize("m,heads,n,k", [(8, 4, 512, 128), (16, 4, 128, 256), (8, 4, 128, 512)])
def test_small_matrix_per_head_no_further_from_64_bits_than_chains_of_multiply_adds(m, heads, n, k):
    """Sums whose second half takes the first away again: what is left is the error of the sums alone."""
    import numpy as np
    o = ops()
    g = torch.Generator().manual_seed(k)
    a, w = torch.randn(m, heads, k // 2, generator=g).bfloat16(), torch.randn(heads, n, k // 2, generator=g).bfloat16()
    a, w = torch.cat([a, -a], 2), torch.cat([w, w], 2)
    out = torch.empty(m, heads * n, dtype=torch.bfloat16, device=DEV)
    o.batched_linear(a.reshape(m, -1).to(DEV), k, w.to(DEV), out, n)
    x, y = a.float().numpy(), w.float().numpy()
    chain = np.zeros((m, heads, n), dtype=np.float32)
    for i in range(k):  # (a product of two bfloat16 values is exact in float32: a chain of multiply-adds)
        chain += x[:, :, None, i] * y[None, :, :, i]
    assert float(out.double().norm()) <= float(np.linalg.norm(chain.astype(np.float64)))


@pytest.mark.parametrize("inter", [1, 8, 31, 33, 64, 127, 700, 1024, 1025, 4100])
@pytest.mark.parametrize("gated", [0, 1, 8])
@pytest.mark.parametrize("n", [1, 33, 67])
def test_square_of_relu_with_a_gate_for_rows_of_any_length(inter, gated, n):
    """Several short rows a CTA, one long row a CTA and more: every value of every row, none beside it."""
    o = ops()
    g = torch.Generator().manual_seed(inter + n)
    u = torch.randn(n, inter + gated, generator=g)
    u[0, 0] = math.nan  # (not above zero: nothing)
    want = torch.relu(torch.nan_to_num(u[:, :inter].double(), nan=0.0)).square()
    if gated:
        want = want * torch.sigmoid(u[:, inter:inter + 1].double())
    for dtype, tol in ((torch.float32, 1e-6), (torch.bfloat16, 2.0 ** -8)):
        kept = torch.full((n + 2, inter), 7.0, dtype=dtype, device=DEV)
        o.relu2_gate(u.to(DEV), kept[:n])
        assert torch.allclose(kept[:n].cpu().double(), want, rtol=tol, atol=1e-7) and (kept[n:] == 7.0).all()
