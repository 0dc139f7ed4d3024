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
