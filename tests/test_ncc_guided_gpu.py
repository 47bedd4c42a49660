"""Guided NCC (csrc/ncc_guided.cuh) against the oracle, bit-exact, where its
blocks, disparity chunks and image edges can go wrong: ranges of one to all
disparities (several chunks of 32), empty blocks, ragged blocks at the right
and lower edge, every window, minimum disparities."""
import numpy as np
import pytest
import torch

from conftest import to_dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,H,D,r,dmin,spread,holes", [
    (64, 32, 16, 5, 0, 0, 0.0),       # whole blocks, ranges of 9
    (250, 37, 200, 5, 0, 199, 0.2),   # every disparity: 7 chunks; ragged blocks
    (250, 37, 200, 2, 3, 90, 0.5),
    (161, 50, 256, 4, 0, 255, 0.9),   # most disparities; many empty blocks
    (49, 17, 40, 5, 11, 20, 0.3),     # a block of one row and of one column
    (33, 40, 33, 4, 2, 32, 0.0),      # one disparity past a chunk
    (40, 16, 8, 5, 60, 8, 0.0),       # minimum disparity beyond the width
])
def test_guided_ncc_is_bit_exact(ct, oracle, cuda, W, H, D, r, dmin, spread, holes):
    L, R, _, _ = ct.synth_pair(2, W + D + r, W, H, max(1, min(W, D + dmin) - 1))
    L[3:12, 5:30] = 90  # flat: the zero-score rule
    g = np.random.default_rng(W + H)
    coarse = dmin + g.integers(0, D) + g.integers(-spread, spread + 1, (H, W))  # scale 1: a hint a pixel
    coarse = np.clip(coarse, 0, dmin + D - 1).astype(np.int16)
    coarse[g.random((H, W)) < holes] = -1
    coarse[:16, :16] = -1
    m = ct.BlockMatcherNCC()
    m.configure(0, W, H, D, radius=r, disp_min=dmin)
    out, score = ct.alloc_image(H, W, torch.int16, cuda), ct.alloc_image(H, W, torch.float32, cuda)
    m.process(out, to_dev(L, cuda), to_dev(R, cuda), score=score,
              disp_init=to_dev(oracle.to_u16(coarse).view(np.int16), cuda))
    d, s32, _ = oracle.match_ncc_guided(L, R, D, coarse, r, dmin=dmin)
    np.testing.assert_array_equal(out.cpu().numpy().view(np.uint16), oracle.to_u16(d))
    got = score.cpu().numpy()
    np.testing.assert_array_equal(got[d >= 0], s32[d >= 0])
    assert not got[d < 0].any()
    assert m.device_status() == 0
