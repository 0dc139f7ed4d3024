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
