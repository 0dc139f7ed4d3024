"""Several tensors copied or cleared in one launch."""
import pytest
import torch

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


@pytest.mark.parametrize("sizes", [[1], [0, 5, 16], [3, 4096, 70001, 8], [17] * 40, [1 << 20, 1, 1 << 18]])
def test_pieces_are_copied_cleared_and_taken_back(sizes):
    """Whole words of 16, 4 and 1 bytes, empty pieces, more than a launch takes; what lies around them stays."""
    from nnis_b200.csrc import ops
    g = torch.Generator().manual_seed(len(sizes))
    room = [torch.randint(0, 255, (n + 32,), dtype=torch.uint8, generator=g).to(DEV) for n in sizes]
    for shift in (0, 4, 1):
        held = [r.clone() for r in room]
        parts = [h[shift + 8:shift + 8 + n] for h, n in zip(held, sizes)]
        want = [p.clone() for p in parts]
        pieces = ops.Pieces(parts)
        kept = pieces.copies()
        assert all(torch.equal(a, b) for a, b in zip(kept, want))
        pieces.clear()
        for r, h, n in zip(room, held, sizes):
            expect = r.clone()
            expect[shift + 8:shift + 8 + n] = 0
            assert torch.equal(h, expect)
        pieces.take_back(kept)
        assert all(torch.equal(r, h) for r, h in zip(room, held))
