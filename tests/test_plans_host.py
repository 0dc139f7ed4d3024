"""Work lists that the host makes for kernels: checked without a GPU."""
import math


def test_prompt_attention_plan_cuts_tiles_without_empty_chunks():
    from nnis_b200.csrc import ops as o
    for counts, starts, window in [([2048], [0], 0), ([700, 3], [100, 0], 0), ([5000], [0], 300),
                                   ([129], [64 * 37 + 5], 0)]:
        for sms in (1, 148, 10 ** 6):
            units, slots = o.prefill_tc_plan(counts, starts, window, 9, sms)
            per_tile = {}
            for s, q0, z, slot in units.tolist():
                per_tile.setdefault((s, q0), []).append((z & 0xffff, z >> 16, slot))
            assert sorted(per_tile) == sorted((i, q0) for i, c in enumerate(counts) for q0 in range(0, c, 128))
            used = 0
            for (s, q0), chunks in per_tile.items():
                n = chunks[0][1]
                assert sorted(c for c, _, _ in chunks) == list(range(n)) and all(k == n for _, k, _ in chunks)
                rows = min(128, counts[s] - q0)
                pos0 = starts[s] + q0
                lo = max(0, pos0 - window + 1) if window else 0
                pages = (pos0 + rows - 1) // 64 - lo // 64 + 1
                assert (n - 1) * (-(-pages // n)) < pages
                used += n if n > 1 else 0
                if n > 1:  # the chunks of a tile share its first scratch slot; tiles do not overlap
                    assert len({slot for _, _, slot in chunks}) == 1
            assert used == slots
            firsts = sorted((chunks[0][2], chunks[0][1]) for chunks in per_tile.values() if chunks[0][1] > 1)
            assert all(a[0] + a[1] <= b[0] for a, b in zip(firsts, firsts[1:]))


def test_decode_attention_slices_fill_waves():
    """The slices of a decode step's key range: as many CTAs as run together, fewer
    waves before shorter slices, never below 256 keys a slice."""
    import torch
    from nnis_b200.engine.context import StepContext
    empty = torch.zeros(0, dtype=torch.int32)

    def pick(ctas, context, resident=444):
        ctx = StepContext(n_tokens=0, n_seqs=0, tokens=empty, token_pos=empty, token_seq=empty,
                          seq_slots=empty, page_tables=[], workspace=None, decode=True, max_context=context)
        return ctx.decode_splits(ctas, resident, 64)

    # one wave where the groups divide the resident CTAs: batch 8, 16, 32, 64 of three kv heads
    assert [pick(c, 4096) for c in (24, 48, 96, 192)] == [16, 9, 4, 2]
    # a wave that would stay 42 % empty is cut further: 256 groups take three slices, two waves
    assert pick(256, 4096) == 3
    # more groups than resident CTAs: no slices at all
    assert pick(2048, 4096) == 1
    for ctas in (1, 3, 40, 100, 443, 445, 5000):
        for context in (1, 64, 300, 4096, 8192, 100000):
            s = pick(ctas, context)
            assert 1 <= s <= 64 and (s - 1) * 256 < max(context, 1)
    # short contexts are not cut
    assert pick(3, 200) == 1 and pick(3, 512) == 2


def test_prompt_attention_plan_takes_the_shortest_chunks_that_fit_one_wave():
    """One prompt of 2,048 tokens, nine heads, 148 SMs: chunks of 12 pages are the longest
    that give enough CTAs, chunks of 11 the shortest with which two CTAs to an SM still hold
    them all (a CTA walks its pages one after another: the longest chunk ends last)."""
    from nnis_b200.csrc import ops as o
    units, _ = o.prefill_tc_plan([2048], [0], 0, 9, 148)
    chunks = {}
    for s, q0, z, slot in units.tolist():
        chunks[q0] = z >> 16
    assert len(units) * 9 <= 2 * 148 and len(units) == 32
    assert chunks[2048 - 128] == 3 and chunks[0] == 1 and chunks[128 * 10] == 2  # 32, 2 and 22 pages
    # 4,096 tokens: a tile a CTA fills a wave; 1,024: chunks of eight pages as before
    assert len(o.prefill_tc_plan([4096], [0], 0, 9, 148)[0]) == 32
    assert max(z >> 16 for _, _, z, _ in o.prefill_tc_plan([1024], [0], 0, 9, 148)[0].tolist()) == 2


def test_bench_sums_a_traced_step_per_kernel():
    import importlib.util
    import os
    spec = importlib.util.spec_from_file_location("bench", os.path.join(os.path.dirname(__file__), "..", "bench.py"))
    bench = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(bench)
    big = 1 << 62
    # per launch: begin, end, first and last past the wait, marks
    rows = [[1000, 4000, 1500, 2000, big, 0, big, 0], [3500, 9000, 4500, 5000, big, 0, big, 0],
            [8000, 9500, big, 0, big, 0, big, 0]]
    got = bench.kernel_times(["a", "b", "a"], rows)
    assert got["a"] == {"launches": 2, "us": 3.5} and got["b"] == {"launches": 1, "us": 4.0}
    assert got["step"] == {"launches": 3, "us": 8.5}


def test_a_begun_norm_is_handed_on_once_and_only_to_the_block_that_owns_it():
    """What a part leaves of a norm in the step's context: taken by the norm it names,
    dropped when another norm asks first, never seen twice; and the prenorm arrangement
    offers a norm only where the part after it says it takes it."""
    import torch
    from nnis_b200.engine.context import StepContext
    from nnis_b200.parts.base import SharedNorm, begin_norm
    from nnis_b200.parts.block import PreNormBlock
    empty = torch.zeros(0, dtype=torch.int32)

    class Space:
        def get(self, name, shape, dtype):
            return torch.zeros(shape, dtype=dtype)

    ctx = StepContext(n_tokens=0, n_seqs=0, tokens=empty, token_pos=empty, token_seq=empty,
                      seq_slots=empty, page_tables=[], workspace=Space(), decode=True, max_context=1)

    class Norm:
        kind = "rmsnorm"
        weight = torch.ones(16)
        eps = 1e-5

    a, b = Norm(), Norm()
    assert begin_norm(ctx, 3, 16) is None and ctx.shared_norm is None  # no block asked for it
    ctx.emit_for = a
    x, weight, shares = begin_norm(ctx, 3, 16)
    assert x.shape == (3, 16) and x.dtype == torch.bfloat16 and shares.shape == (3, 2) and weight is a.weight
    assert isinstance(ctx.shared_norm, SharedNorm)
    assert ctx.take_shared_norm(a).x is x and ctx.take_shared_norm(a) is None
    begin_norm(ctx, 3, 16)
    assert ctx.take_shared_norm(b) is None and ctx.take_shared_norm(a) is None  # dropped, not kept
    assert begin_norm(ctx, 3, 12) is None  # a width that is no multiple of eight
    other = Norm()
    other.kind = "layernorm"
    ctx.emit_for = other
    assert begin_norm(ctx, 3, 16) is None

    # the arrangement: which norm each part is told about, and what reaches the parts
    calls = []

    class Mixer:
        def forward(self, x, ctx, residual, cache):
            calls.append(("mixer", ctx.emit_for))

    class SharingFfn:
        def shares_norm(self, norm, ctx, n):
            return True

        def forward(self, x, ctx, residual):
            calls.append(("ffn", ctx.emit_for))

        def forward_shared(self, begun, residual, ctx):
            calls.append(("ffn shared", begun.norm))

    class PlainNorm(Norm):
        def forward(self, hidden, out, rows=None):
            pass

    block = PreNormBlock.__new__(PreNormBlock)
    block.dtype = torch.bfloat16
    block.mixer_norm, block.ffn_norm = PlainNorm(), PlainNorm()
    block.mixer, block.ffn = Mixer(), SharingFfn()
    ctx.emit_for = None
    ctx.next_norm = a
    hidden = torch.zeros(3, 16)
    assert block.first_shared_norm(ctx, 3) is None  # this mixer takes no begun norm
    block.forward(hidden, ctx, None)
    # the mixer was told of the feed-forward's norm and left nothing: the norm ran whole;
    # the feed-forward was told of the next block's first norm
    assert calls == [("mixer", block.ffn_norm), ("ffn", a)] and ctx.emit_for is None

    class EmittingMixer(Mixer):
        def forward(self, x, ctx, residual, cache):
            begin_norm(ctx, 3, 16)

    calls.clear()
    block.mixer = EmittingMixer()
    block.forward(hidden, ctx, None)
    assert calls == [("ffn shared", block.ffn_norm)] and ctx.shared_norm is None


def test_decode_attention_by_tma_takes_the_longest_slices_that_stay_resident():
    """The slices of the decode attention whose pages are all in shared memory at once, on a
    device of 148 SMs that holds three CTAs of four pages, two of five or six, one of seven or
    eight to an SM (head size 64): four pages; six where four make more CTAs than two to an
    SM; beyond 16 slices, eight or six where those CTAs are all resident; else not this kernel."""
    from nnis_b200.csrc.ops import tma_slices
    fit = lambda pages: 3 if pages <= 4 else 2 if pages <= 6 else 1

    def slices(sequences, pages, kv_heads=3, fixed=0):
        return tma_slices(sequences * kv_heads, pages, 148, 8, fit, fixed)

    # context 4,096 (64 pages): one to six sequences 16 slices of four pages, seven and eight
    # 11 slices of six (two CTAs to an SM), nine 16 of four again (297 CTAs of six pages are one too
    # many for two to an SM; 432 of four fit three to an SM), ten and more none
    assert [slices(n, 64) for n in (1, 2, 6, 7, 8, 9)] == [16, 16, 16, 11, 11, 16]
    assert slices(10, 64) == 0 and slices(64, 64) == 0
    # short contexts: one slice, many sequences
    assert slices(1, 1) == 1 and slices(40, 4) == 1 and slices(200, 4) == 0
    # beyond 16 slices of four pages: eight pages one to an SM, six pages two to an SM
    assert slices(1, 128) == 16 and slices(3, 128) == 16 and slices(4, 128) == 22
    assert slices(1, 256) == 32 and slices(2, 256) == 43 and slices(3, 256) == 0
    assert slices(1, 384) == 48 and slices(1, 512) == 86 and slices(2, 512) == 0
    # never more than 128 slices, never more than eight pages a slice
    assert slices(1, 1024) == 0 and slices(1, 1000, kv_heads=1) == 125 and slices(1, 1025, kv_heads=1) == 0
    # a fixed slice length is taken if its CTAs are resident
    assert slices(8, 64, fixed=4) == 16 and slices(8, 64, fixed=8) == 0 and slices(2, 64, fixed=8) == 8
    for n in (1, 2, 3, 5, 8, 13, 40):
        for pages in (1, 3, 16, 17, 63, 64, 65, 100, 128, 129, 255, 256, 400, 512, 700):
            s = slices(n, pages)
            if s:
                per = -(-pages // s)
                assert 1 <= s <= 128 and per <= 8 and s * per >= pages
                assert n * 3 * s <= 148 * fit(per)


def _ops_with_the_library():
    """The kernels' library holds the rules of which kernel takes which product as plain host
    functions; they need no GPU, only the library (built with nvcc at first use)."""
    import pytest
    from nnis_b200.csrc import ops
    try:
        ops._lib()
    except Exception as e:  # no compiler here
        pytest.skip(f"the kernels' library is not built here: {e}")
    return ops


def test_which_kernel_takes_the_projections_of_a_decode_step():
    """On 148 SMs, for the SmolLM2 shapes: 2 the kernel over tiles of rows, 1 the kernel whose
    CTAs hold all rows, 0 neither (norm kernel and tensor-core product); and where the norm
    before QKV and before gate/up can be shared out between the projections around it."""
    o = _ops_with_the_library()

    def plans(H, inter, nq, nkv, d, m):
        qkv = (nq + 2 * nkv) * d
        return dict(qkv=o.gemv_kind(m, qkv, H, o.EPI_QKV, None, True),
                    qkv_shares=o.gemv_kind(m, qkv, H, o.EPI_QKV, shared_norm=True) == 2,
                    out=o.gemv_kind(m, H, nq * d, o.EPI_ADD_F32),
                    gate_up=o.gemv_kind(m, 2 * inter, H, o.EPI_GATED, None, True),
                    gate_up_shares=o.gemv_kind(m, 2 * inter, H, o.EPI_GATED, shared_norm=True) == 2,
                    down=o.gemv_kind(m, H, inter, o.EPI_ADD_F32), down_slices=o.gemv_slices(m, H, inter))

    small, middle, large = (576, 1536, 9, 3, 64), (960, 2560, 15, 5, 64), (2048, 8192, 32, 32, 64)
    # the benchmark's shape: everything over tiles of rows up to 64 rows, both norms shared
    for m in (1, 8, 16, 48, 64):
        assert plans(*small, m) == dict(qkv=2, qkv_shares=True, out=2, gate_up=2, gate_up_shares=True,
                                        down=2, down_slices=1), m
    # at 128 rows gate/up has more CTAs than are resident at once
    p = plans(*small, 128)
    assert (p["qkv"], p["out"], p["down"], p["gate_up"], p["gate_up_shares"]) == (2, 2, 2, 0, False)
    # the 360M shape: the same up to 16 rows, its down projection in two slices of K;
    # from 48 rows on gate/up (640 units) leaves the kernel over tiles of rows and shares no norm
    for m in (1, 8, 16):
        assert plans(*middle, m) == dict(qkv=2, qkv_shares=True, out=2, gate_up=2, gate_up_shares=True,
                                         down=2, down_slices=2), m
    for m in (48, 64):
        p = plans(*middle, m)
        assert (p["qkv"], p["qkv_shares"], p["gate_up"], p["gate_up_shares"]) == (2, True, 1, False), m
    # the 1.7B shape: rows of 2,048 are longer than a warp's share of x in registers, so the
    # norm stays in the prologue of the kernel whose CTAs hold all rows, and nothing is shared;
    # the down projection (K = 8,192) runs in four slices of K
    for m in (1, 8, 16):
        p = plans(*large, m)
        assert (p["qkv"], p["qkv_shares"], p["gate_up"], p["gate_up_shares"]) == (1, False, 1, False), m
        assert (p["out"], p["down"], p["down_slices"]) == (2, 1, 4), m
    # what no decode kernel takes: more than 128 rows, K off a multiple of 16, N off a multiple of 8
    assert o.gemv_kind(129, 576, 576, o.EPI_ADD_F32) == 0 and o.gemv_kind(8, 576, 568, o.EPI_ADD_F32) == 0
    assert o.gemv_kind(8, 572, 576, o.EPI_ADD_F32) == 0
    # a shared norm ends only in the QKV and the gated epilogue
    assert o.gemv_kind(8, 576, 576, o.EPI_STORE, shared_norm=True) == 0
    # the adding tensor-core product cuts a long K among CTAs only where tiles are few
    assert o.gemm_tc_splits(64, 2048, 8192)[0] == 4 and o.gemm_tc_splits(2048, 576, 1536)[0] == 1


def test_adding_projections_share_k_in_one_launch_where_two_launches_are_not_faster():
    """Two parts of more CTAs than two an SM leave the product to two launches; more parts never do."""
    from nnis_b200.csrc import ops as o
    for m, n, k, one_launch in ((8, 2048, 2048, True), (8, 4096, 3072, True), (8, 6144, 3072, False), (1, 6144, 2048, False),
                                (17, 2048, 3072, True), (17, 3072, 1792, False), (64, 1024, 2560, True), (64, 1536, 2048, False),
                                (64, 2048, 3072, False), (64, 2048, 8192, True), (32, 4096, 4096, True), (8, 6144, 4096, True)):
        floats, tiles = o.gemv_split_scratch(m, n, k)
        assert (floats > 0) == (tiles > 0) == one_launch, (m, n, k)
        assert o.gemv_slices(m, n, k) >= 2


def test_which_retention_prompts_work_their_chunks_side_by_side(monkeypatch):
    from nnis_b200.csrc import ops as o
    side = lambda counts, heads=8, dim=128, vdim=256: o.retention_side_by_side(counts, heads, dim, vdim, 148)
    assert side([300]) and side([200, 200]) and side([2048]) and side([100] * 16) and not side([100] * 16, heads=4)
    assert not side([150]) and not side([255]) and not side([90] * 4) and not side([128] * 4) and not side([60] * 4)
    assert not side([2048], dim=48)
    for off in (0, 100):  # (no multiple of 32)
        monkeypatch.setattr(o, "RETENTION_SEGMENT", off)
        assert not side([2048]) and not o.retention_takes_chunks(128)


def test_launches_of_retention_side_by_side_are_those_of_its_waves():
    """Four kernels a wave and the gate: waves of whole pairs where chunks go by pairs, of chunks where not."""
    from nnis_b200.csrc import ops as o
    launches = lambda chunks, seqs, dim, vdim, wave, heads=8: o.retention_launches(chunks, seqs, heads, dim, vdim, wave)
    assert launches(32, 1, 128, 256, 32) == 5 and launches(100, 1, 128, 256, 3) == 4 * 50 + 1 and launches(100, 1, 128, 8, 2) == 4 * 50 + 1
    assert launches(100, 1, 128, 256, 1) == 401 and launches(100, 1, 128, 250, 3) == 4 * 34 + 1 and launches(100, 1, 32, 64, 3) == 4 * 34 + 1
    assert launches(48, 16, 64, 256, 10) == 4 * 7 + 1  # 32 pairs at most, five at a time
    # small heads: by pairs where sequences are long and many CTAs come of them
    assert launches(63, 1, 64, 64, 6) == 4 * 11 + 1 and launches(12, 1, 64, 64, 6) == 4 * 2 + 1 and launches(48, 16, 64, 64, 10) == 4 * 5 + 1


def test_chunks_of_recurrent_layers_keep_their_scratch_within_its_bound():
    """As many chunks at a time as the scratch holds, one at least; all of them as long as they fit."""
    from nnis_b200.csrc import ops as o
    assert o.retention_wave(32, 8, 128, 256) == 32   # 2,048 tokens
    for chunks in (1, 56, 57, 256, 4096):
        a, b = o.retention_scratch(chunks, 8, 128, 256)
        wave = o.retention_wave(chunks, 8, 128, 256)
        assert 1 <= wave <= chunks and (a, b) == (wave * 8 * 64 * (3 * 128 + 256), wave * 8 * 128 * 256)
        assert 4 * (a + b) <= o.RETENTION_SCRATCH
    assert o.retention_wave(9, 4096, 256, 1024) == 1  # (more than the bound for a single one)


def test_chunks_of_the_delta_rule_keep_their_scratch_within_its_bound():
    from nnis_b200.csrc import ops as o
    assert o.delta_wave(52, 32, 16, 128, 128) == 52   # 3,300 tokens
    wave = o.delta_wave(4096, 32, 16, 128, 128)
    asked = lambda n: sum(math.prod(shape) * dtype.itemsize for _, shape, dtype in o.delta_scratch(n, 32, 16, 128, 128))
    assert asked(wave) <= o.DELTA_SCRATCH < 1 << 30 and asked(wave + 1) > o.DELTA_SCRATCH and 64 * wave > 8500
    assert o.delta_wave(9, 4096, 4096, 128, 512) >= 1


def test_which_prompts_of_the_matrix_memory_go_by_pairs_of_chunks():
    """Not short ones, not heads of 64 x 64, not many sequences of one chunk with small heads."""
    from nnis_b200.csrc import ops as o
    pairs = lambda counts, heads=8, dim=128, vdim=256: o.memory_by_pairs(counts, heads, dim, vdim, 148)
    assert pairs([2000]) and pairs([40]) and pairs([33]) and pairs([1500, 1500, 701]) and pairs([300, 1, 17])
    assert not pairs([1]) and not pairs([32]) and not pairs([16, 24, 30]) and pairs([64]) and pairs([66])
    assert pairs([24] * 16) and not pairs([24] * 8) and not pairs([24] * 64, vdim=128)
    assert not pairs([2000], dim=64, vdim=64) and pairs([2000], dim=64, vdim=72) and pairs([2000], vdim=8)
    assert not pairs([2000], dim=96) and not pairs([2000], vdim=100)
    assert not pairs([64] * 64, dim=64, vdim=128) and pairs([64] * 64, dim=64, vdim=136) and pairs([100] * 64, dim=64, vdim=128)
    assert pairs([64] * 16, vdim=64) and not pairs([64] * 19, vdim=64)


def test_float32_prompts_take_tiles_where_these_pay():
    """Enough queries to a tile, or a long chain of keys on an empty device; the counts behind the rule are those of the
    tiles and of the keys that the queries see."""
    from nnis_b200.csrc import ops as o
    pays = o.attention_tile_f32_pays
    assert pays([509, 131, 384], [0, 0, 0], 0, 9) and pays([64], [0], 0, 9) and pays([1] * 8, [2000] * 8, 0, 9)
    assert not pays([1] * 64, [500] * 64, 0, 9) and not pays([8], [64], 0, 9) and not pays([8] * 64, [0] * 64, 0, 9)
    assert pays([500] + [1] * 15, [0] + [2000] * 15, 0, 16) and not pays([4] * 64, [2000] * 64, 0, 16)
    # a window of 50 keys: the far past counts for nothing
    assert pays([64] * 64, [4000] * 64, 50, 9) == pays([64] * 64, [64 * 50] * 64, 50, 9)
    assert not pays([1, 1, 2], [4000, 3000, 2000], 50, 9) and pays([1, 1, 2], [4000, 3000, 2000], 0, 9)
    for window in (0, 1, 7, 64, 100):  # where the first part is nothing: pages x heads against keys x heads / 500
        for c, st in ((1, 0), (20, 3), (64, 0), (65, 40), (100, 20)):
            keys = sum(min(st + q + 1, window or 10 ** 9) for q in range(c))
            tiles = [(st + q0, st + min(q0 + 64, c) - 1) for q0 in range(0, c, 64)]
            pages = sum(b // 64 - (max(0, a - window + 1) if window else 0) // 64 + 1 for a, b in tiles)
            assert pays([c], [st], window, 1000) == (pages * 1000 <= keys * 2)


def test_which_float32_products_run_on_the_tensor_cores():
    """More rows than a decode step's kernel takes, whole groups of eight columns, 32-byte boundaries; a K below 128 only with a
    large output."""
    import torch
    from nnis_b200.csrc import ops as o

    def pays(m, n, k, off=0):
        at = lambda rows: torch.empty(rows * k + 8)[off:off + rows * k].view(rows, k)
        a, w = at(m), at(n)
        assert off or a.data_ptr() % 32 == 0 == w.data_ptr() % 32
        return o.gemm_split_f32_pays(a, w)
    assert pays(17, 576, 576) and pays(17, 8, 128) and pays(512, 3072, 64) and pays(100, 8192, 96)
    assert not pays(16, 576, 576) and not pays(17, 576, 580) and not pays(17, 576, 576, 1)
    assert not pays(64, 3072, 64) and not pays(512, 576, 96) and not pays(64, 12000, 120)


def test_which_kernel_takes_a_float32_prompt_step_of_heads_of_64(monkeypatch):
    """Tiles of 128 queries on the tensor cores, tiles of 64 for many prompts of one page, a warp a query for few short ones;
    a step is planned once for all layers with its window and heads."""
    import torch
    from nnis_b200.csrc import ops as o
    from nnis_b200.parts.attention import Attention
    monkeypatch.setattr(o, "sm_count", lambda device: 148)
    monkeypatch.setattr(o, "TC_ATTENTION", 1)

    def kinds(counts, starts=None, heads=9, window=0):
        part = Attention.__new__(Attention)
        part.dtype, part.heads, part.head_dim, part.window, part.device = torch.float32, heads, 64, window, "cpu"
        starts = starts or [0] * len(counts)
        tables = part.step_tables(counts, starts)
        assert part.step_tables(counts, starts, tuple(tables)) == {}
        tiles = [v for k, v in tables.items() if k == part._tile_f32_name()]
        if tiles:
            assert sorted(tiles[0].tolist()) == [[i, q0] for i, c in enumerate(counts) for q0 in range(0, c, 64)]
        units = any(k.endswith("/units") for k in tables)
        assert not (units and tiles)
        return "tcgen05" if units else "tiles" if tiles else "warps"
    assert kinds([1024]) == kinds([64]) == kinds([100] * 10) == kinds([64] * 8) == kinds([17], [500]) == kinds([65] * 40) == "tcgen05"
    assert kinds([64] * 40) == kinds([50] * 40) == kinds([40] * 8, heads=32) == kinds([64] * 40, heads=4) == "tiles"
    assert kinds([17]) == kinds([8] * 64) == kinds([300], window=30) == kinds([20] * 40, heads=32) == "warps"


def test_slices_of_the_float32_prompt_attention_keep_their_scratch_within_its_bound():
    """Records are as many as the most slices of any tile for every row of the step; long steps are cut less, or not."""
    from nnis_b200.csrc import ops as o
    for heads in (1, 9, 32, 128):
        for counts, starts in (([65536], [0]), ([16384], [49152]), ([8192], [0]), ([8192], [8192]), ([1] * 3000 + [128], [0] * 3000 + [60000]),
                               ([4096] * 8, [0] * 8), ([30000], [0]), ([1024], [0])):
            for sms in (40, 148, 1000):
                plan = o.attention_split_f32_plan(counts, starts, 0, heads, sms)
                if plan is not None and plan[1] > 1:
                    assert 4 * sum(counts) * heads * plan[1] * (64 + 2) <= o.SPLIT_F32_SCRATCH <= 1 << 28
    assert o.attention_split_f32_plan([1024], [0], 0, 9, 148)[1] > 1 and o.attention_split_f32_plan([65536], [0], 0, 9, 148)[1] == 1


def test_units_of_the_float32_prompt_attention_cover_every_tile_once():
    import random
    from nnis_b200.csrc import ops as o
    rng = random.Random(5)
    for _ in range(300):
        n = rng.randint(1, 6)
        counts, starts = [rng.choice((1, 17, 128, 129, 700)) for _ in range(n)], [rng.choice((0, 5, 64, 900)) for _ in range(n)]
        window = rng.choice((0, 0, 1, 100))
        plan = o.attention_split_f32_plan(counts, starts, window, rng.choice((1, 9, 32)), rng.choice((1, 40, 148)))
        if plan is None:
            continue
        units, slices = plan
        seen = {}
        for i, q0, z, k in units.tolist():
            first, last = starts[i] + q0, starts[i] + min(q0 + 128, counts[i]) - 1
            pages = last // 64 - (max(0, first - window + 1) if window else 0) // 64 + 1
            per = -(-pages // k)
            assert 0 <= z < k <= slices and (z * per < pages)  # (no slice is empty)
            seen.setdefault((i, q0), []).append((z, k))
        assert set(seen) == {(i, q0) for i, c in enumerate(counts) for q0 in range(0, c, 128)}
        for parts in seen.values():
            assert sorted(z for z, _ in parts) == list(range(parts[0][1])) and len({k for _, k in parts}) == 1
        assert max(k for _, _, _, k in units.tolist()) == slices


def _latent_decode_source():
    import os
    from nnis_b200 import csrc
    with open(os.path.join(os.path.dirname(csrc.__file__), "attention_latent_decode.cu")) as f:
        return f.read()


def test_stores_into_the_latent_ring_are_fenced_before_the_copies_over_them():
    """Ordinary stores and bulk copies to the same shared memory are ordered by a proxy fence of the storing threads alone; no
    result shows that it is missing, so the kernel's text is looked at: from the zeroed rows to the next barrier."""
    text = _latent_decode_source()
    stores = text[text.index("if (row < r0 || row >= r1) *at ="):]
    assert "fence.proxy.async.shared::cta" in stores[:stores.index("__syncthreads()")]


def test_padding_rows_of_latent_decode_wait_for_the_kernel_ahead_too():
    """What comes after a kernel counts on all before it being over; a grid of padding rows alone (the run before a capture)
    that returns at once would break the chain, and no result shows it."""
    text = _latent_decode_source()
    padding = text[text.index("if (pos < 0)"):]
    assert "pdl_wait();" in padding[:padding.index("return;")]
