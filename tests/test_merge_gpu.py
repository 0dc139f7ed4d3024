"""The merge of split attention's records at the edges of its forms."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("rows,d,n", [(1, 66, 9), (1184, 96, 16), (1185, 96, 16), (128, 512, 16), (3, 600, 13), (296, 512, 8), (297, 512, 8),
                                      (5, 258, 1), (7, 512, 17), (4, 128, 64), (9, 97, 12), (148, 320, 8), (149, 320, 8), (445, 512, 9),
                                      (593, 256, 12), (889, 136, 9), (1037, 256, 9), (1184, 384, 9), (2, 1024, 16), (297, 600, 9), (5, 1024, 8)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float32])
def test_slices_meet_as_in_64_bits(rows, d, n, dtype):
    from nnis_b200.csrc import ops
    g = torch.Generator().manual_seed(rows + d + n)
    rec = torch.randn(rows, n, d + 2, generator=g)
    rec[..., 0] *= 8
    rec[..., 1] = rec[..., 1].abs() + 0.1
    empty = torch.rand(rows, n, generator=g) < 0.3
    empty[0] = True  # (a row whose slices all hold nothing is zero)
    rec[..., 1][empty] = 0
    rec[..., 2:][empty] = float("nan")  # (what such a slice holds is never written, and never added)
    m, l, v = rec[..., 0].double(), rec[..., 1].double(), rec[..., 2:].double()
    w = torch.where(empty, 0.0, (m - m.masked_fill(empty, -1e30).amax(1, keepdim=True)).clamp(max=0).exp())
    want = (w[..., None] * v.masked_fill(empty[..., None], 0)).sum(1) / (w * l).sum(1, keepdim=True).clamp(min=1e-300)
    part, out = rec.to(DEV), torch.full((rows, d), 9.0, dtype=dtype, device=DEV)
    lib = ops._lib()
    merge = lib.nnis_attention_merge_bf16 if dtype == torch.bfloat16 else lib.nnis_attention_merge_f32
    code = merge(ops._ptr(part), ops._ptr(out), ctypes.c_longlong(rows), d, n, ops._stream())
    assert code == 0
    # bfloat16 rounds at 2^-9; exponentials and up to 64 float32 sums stay within 2^-17 of the sizes they add
    size = (w[..., None] * v.masked_fill(empty[..., None], 0).abs()).sum(1) / (w * l).sum(1, keepdim=True).clamp(min=1e-300)
    assert ((out.cpu().double() - want).abs() <= want.abs() * (2**-8 if dtype == torch.bfloat16 else 0) + size * 2**-17).all()
