"""Absolute-difference matchers on four-byte differences: every alignment of
the match bytes (minimum disparity mod 4), both directions, every window, on
full-contrast noise (the largest window sums), and the sub-pixel step where a
tile's winners span the whole range of 256 disparities. Bit-exact."""
import numpy as np
import pytest
import torch

from conftest import to_dev

pytestmark = pytest.mark.gpu


def noise(seed, W, H):
    g = np.random.default_rng(seed)
    return [np.where(g.random((H, W)) < 0.5, 0, 255).astype(np.uint8) for _ in range(2)]


@pytest.mark.parametrize("dmin", [0, 1, 2, 3])
@pytest.mark.parametrize("lr", [True, False])
@pytest.mark.parametrize("r", [1, 2, 3, 4])
def test_sad_alignments(ct, oracle, cuda, r, lr, dmin):
    W, H, D = 261, 45, 67
    L, R = noise(16 * r + 4 * lr + dmin, W, H)
    m = ct.BlockMatcherSAD1()
    m.configure(0, W, H, D, radius=r, left_to_right=lr, disp_min=dmin)
    out = ct.alloc_image(H, W, torch.int16, cuda)
    m.process(out, to_dev(L, cuda), to_dev(R, cuda))
    torch.cuda.synchronize()
    want, _ = oracle.match_sad(L, R, D, r, lr, dmin=dmin)
    np.testing.assert_array_equal(out.cpu().numpy().view(np.uint16), oracle.to_u16(want))


@pytest.mark.parametrize("W,H,D,dmin", [(419, 40, 256, 0), (419, 40, 256, 1), (130, 33, 18, 2), (117, 29, 61, 3)])
def test_aw_alignments(ct, oracle, cuda, W, H, D, dmin):
    L, R = noise(W + D + dmin, W, H)
    m = ct.BlockMatcherAW()
    m.configure(0, W, H, D, disp_min=dmin)
    out = ct.alloc_image(H, W, torch.float32, cuda)
    m.process(out, to_dev(L, cuda), to_dev(R, cuda))
    torch.cuda.synchronize()
    _, _, s32, _ = oracle.match_aw(L, R, D, dmin=dmin)
    np.testing.assert_array_equal(out.cpu().numpy(), s32)
