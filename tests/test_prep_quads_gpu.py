"""Rotations and head preparation by fours of values, against the kernels that take any layout."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def off(t):
    """The same values from a row that starts one value later in memory: only the general kernel takes it."""
    room = torch.empty(t.numel() + 1, dtype=t.dtype, device=t.device)
    out = room[1:].view(t.shape)
    out.copy_(t)
    return out


# (multiply-adds contracted otherwise: a rounding of float32, or of the bfloat16 stored)
BOUND = {torch.float32: 2e-6, torch.bfloat16: 2e-2}


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("heads,length,dims,pairing", [(3, 16, 8, "half"), (1, 64, 64, "half"), (5, 12, 12, "neighbours"),
                                                       (16, 72, 64, "neighbours"), (2, 8, 0, "half"), (1, 264, 256, "half")])
@pytest.mark.parametrize("n", [3, 70, 2371])  # (the last by fours whatever the heads)
def test_parts_of_heads_turned_by_fours(dtype, heads, length, dims, pairing, n):
    from nnis_b200.csrc import ops
    g = torch.Generator().manual_seed(heads + length + n)
    src = torch.randn(n, heads * (length + 8), generator=g).to(dtype).to(DEV)
    pos = torch.randint(-1, 4000, (n,), dtype=torch.int32, generator=g).to(DEV)
    freq = (torch.rand(max(dims // 2, 1), generator=g)).to(DEV)
    got, want = torch.zeros(n, heads * (length + 4), dtype=dtype, device=DEV), off(torch.zeros(n, heads * (length + 4), dtype=dtype, device=DEV))
    for x, dst in ((src, got), (off(src), want)):
        ops.rope_part(x, length + 8, 4, dst, length + 4, 4, pos, freq, heads, length, dims, pairing=pairing)
    assert (got.float() - want.float()).abs().max() <= BOUND[dtype]
    assert got.view(n, heads, -1)[..., :4].abs().max() == 0


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H,G,dk,dv,rot,gated,normed", [(16, 4, 64, 64, 64, False, False), (2, 1, 128, 64, 32, True, True),
                                                        (4, 2, 4, 8, 2, True, False), (8, 0, 64, 64, 64, False, True), (3, 3, 260, 4, 256, False, True)])
@pytest.mark.parametrize("n", [1, 71, 447])  # (the last by fours whatever the rows)
def test_heads_prepared_by_fours(dtype, H, G, dk, dv, rot, gated, normed, n):
    import ctypes
    from nnis_b200.csrc import ops
    g = torch.Generator().manual_seed(H + dk + n)
    cols = H * dk + G * (dk + dv) + (H if gated else 0)
    a = torch.randn(n, cols, generator=g).to(DEV)
    pos = torch.arange(50, 50 + n, dtype=torch.int32)
    pos[n // 2] = -1 if n > 1 else 50
    pos, seq = pos.to(DEV), torch.zeros(n, dtype=torch.int32, device=DEV)
    pages = -(-(50 + n) // 64)
    table = torch.randperm(pages, generator=g).to(torch.int32)[None].to(DEV)
    freq, wq, wk = torch.rand(rot // 2, generator=g).to(DEV), torch.rand(H * dk, generator=g).to(DEV), torch.rand(max(G, 1) * dk, generator=g).to(DEV)
    out = []
    for x in (a, off(a)):
        q, gate = torch.full((n, H * dk), 9.0, dtype=dtype, device=DEV), torch.full((n, H), 9.0, device=DEV)
        kc, vc = (torch.full((pages, max(G, 1), 64, d), 9.0, dtype=dtype, device=DEV) for d in (dk, dv))
        P = ops._ptr
        code = ops._lib().nnis_qkv_prep(P(x), P(wq) if normed else None, P(wk) if normed and G else None, P(freq), P(pos), P(seq), P(table), pages,
                                        P(q), P(kc), P(vc), P(gate), n, H, G, dk, dv, rot, int(gated), 64, ctypes.c_float(1e-5),
                                        0 if dtype == torch.float32 else 1, ops._stream())
        assert code == 0
        out.append((q, kc, vc, gate))
    for got, want in zip(*out):
        assert (got.float() - want.float()).abs().max() <= BOUND[dtype] * max(1.0, float(want.float().abs().max()))
        assert torch.equal(got == 9.0, want == 9.0)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("nq,nkv,d,rotate", [(9, 3, 64, 1), (2, 0, 8, 1), (1, 1, 136, 1), (0, 2, 16, 0), (4, 4, 128, 0)])
@pytest.mark.parametrize("n", [1, 71, 741])
def test_heads_rotated_and_stored_by_fours(dtype, nq, nkv, d, rotate, n):
    from nnis_b200.csrc import ops
    g = torch.Generator().manual_seed(nq + d + n)
    qkv = torch.randn(n, (nq + 2 * nkv) * d, generator=g).to(dtype).to(DEV)
    pos = torch.arange(50, 50 + n, dtype=torch.int32)
    pos[n // 2] = -1 if n > 1 else 50
    pos, seq = pos.to(DEV), torch.zeros(n, dtype=torch.int32, device=DEV)
    pages = -(-(50 + n) // 64)
    table = torch.randperm(pages, generator=g).to(torch.int32)[None].to(DEV)
    angle = torch.rand(64 * pages, d // 2, generator=g) * 6
    cos, sin, P, out = angle.cos().to(DEV), angle.sin().to(DEV), ops._ptr, []
    for x in (qkv.clone(), off(qkv)):
        kc, vc = (torch.full((pages, max(nkv, 1), 64, d), 9.0, dtype=dtype, device=DEV) for _ in range(2))
        code = ops._lib().nnis_rope_store(P(x), 0 if dtype == torch.float32 else 1, P(pos), P(seq), P(table), pages, P(cos), P(sin), P(kc), P(vc),
                                          n, nq, nkv, d, 64, rotate, ops._stream())
        assert code == 0
        out.append((x, kc, vc))
    for got, want in zip(*out):
        assert (got.float() - want.float()).abs().max() <= BOUND[dtype] * max(1.0, float(want.float().abs().max()))
        assert torch.equal(got == 9.0, want == 9.0)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16])
@pytest.mark.parametrize("H,G,dk,dv,rot,gated,normed", [(16, 4, 64, 64, 64, True, True), (4, 1, 128, 64, 32, False, True),
                                                        (3, 3, 20, 8, 16, False, True), (8, 8, 128, 128, 128, False, False)])
def test_heads_prepared_by_fours_have_the_general_kernels_bits(dtype, H, G, dk, dv, rot, gated, normed):
    """A prompt's layer gives the same whether its rows lie by fours or not: norms sum in one order."""
    import ctypes
    from nnis_b200.csrc import ops
    n = 601
    g = torch.Generator().manual_seed(H + dk)
    a = (torch.randn(n, H * dk + G * (dk + dv) + (H if gated else 0), generator=g) * 3).to(DEV)
    pos, seq = torch.arange(n, dtype=torch.int32, device=DEV), torch.zeros(n, dtype=torch.int32, device=DEV)
    table = torch.randperm(10, generator=g).to(torch.int32)[None].to(DEV)
    freq, wq, wk = torch.rand(rot // 2, generator=g).to(DEV), torch.rand(H * dk, generator=g).to(DEV), torch.rand(G * dk, generator=g).to(DEV)
    out, P = [], ops._ptr
    for x in (a, off(a)):
        q, gate = torch.full((n, H * dk), 9.0, dtype=dtype, device=DEV), torch.full((n, H), 9.0, device=DEV)
        kc, vc = (torch.full((10, G, 64, d), 9.0, dtype=dtype, device=DEV) for d in (dk, dv))
        assert ops._lib().nnis_qkv_prep(P(x), P(wq) if normed else None, P(wk) if normed else None, P(freq), P(pos), P(seq), P(table), 10,
                                        P(q), P(kc), P(vc), P(gate), n, H, G, dk, dv, rot, int(gated), 64, ctypes.c_float(1e-5),
                                        0 if dtype == torch.float32 else 1, ops._stream()) == 0
        out.append((q, kc, vc, gate))
    for got, want in zip(*out):
        assert torch.equal(got, want)
