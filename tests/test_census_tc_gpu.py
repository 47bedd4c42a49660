"""The census matcher's tensor-core pass (csrc/census_tc.cuh) against the
oracle, bit-exact, at the sizes where it can go wrong: one and two tiles a
pair, a strip's last pair with one tile, the most columns a tile has, the
switch to tiles that share their left pixels, strips of few rows, minimum
disparities, and calls that mix it with the CUDA-core pass."""
import numpy as np
import pytest
import torch

from conftest import to_dev

pytestmark = pytest.mark.gpu


def _want(oracle, L, R, D, dmin, dtype):
    lr, _ = oracle.match_census(L, R, D, 2, True, dmin=dmin)
    rl, _ = oracle.match_census(L, R, D, 2, False, dmin=dmin)
    if dtype == torch.int16:
        a, b = oracle.to_u16(lr), oracle.to_u16(rl)
        return a, b, oracle.crosscheck_codes(a, b, 1, True, frame=False)[0]
    ck, _ = oracle.crosscheck(lr, rl, 1, True)
    return oracle.to_u8(lr), oracle.to_u8(rl), oracle.to_u8(np.where(ck == -2, -1, ck))


def _got(t):
    a = t.cpu().numpy()
    return a.view(np.uint16) if a.dtype == np.int16 else a


@pytest.mark.parametrize("W,H,D,dmin,kind,dtype", [
    (8, 8, 48, 0, 1, torch.int16),        # smallest image, most disparities without a pixel
    (160, 96, 64, 0, 1, torch.uint8),
    (128, 21, 113, 0, 1, torch.int16),    # 240 columns with 128 left pixels; strips of a few rows
    (257, 40, 113, 1, 2, torch.int16),    # one pixel past a pair of tiles, odd minimum
    (254, 33, 114, 0, 1, torch.uint8),    # 127 left pixels a tile
    (339, 37, 128, 5, 2, torch.int16),    # a last pair with one tile
    (300, 30, 150, 0, 1, torch.int16),    # about where tiles start to share their left pixels
    (300, 30, 151, 0, 2, torch.int16),
    (129, 29, 200, 3, 2, torch.int16),
    (640, 50, 256, 0, 2, torch.int16),    # all disparities a key has room for
    (201, 64, 254, 0, 3, torch.uint8),
    (400, 140, 96, 40, 1, torch.int16),   # the match columns start left of the image
    (60, 30, 48, 70, 1, torch.int16),     # minimum disparity beyond the width
])
def test_tensor_core_pass_is_bit_exact(ct, oracle, cuda, W, H, D, dmin, kind, dtype):
    L, R, _, _ = ct.synth_pair(kind, 300 + W + D, W, H, max(1, D - 1 + dmin))
    dl, dr = to_dev(L, cuda), to_dev(R, cuda)
    want = _want(oracle, L, R, D, dmin, dtype)
    m = ct.BlockMatcherCensus()
    m.configure(0, W, H, D, disp_min=dmin)
    out = [ct.alloc_image(H, W, dtype, cuda) for _ in range(3)]
    m.process_lr(dl, dr, *out, tol=1)
    for name, o, w in zip(("left", "right", "checked"), out, want):
        np.testing.assert_array_equal(_got(o), w, err_msg=name)
    for o in out:
        o.fill_(77)
    m.process_lr(dl, dr, disp_rl=out[1])     # the right view alone
    m.process(out[0], dl, dr)                # the left view alone
    m.process_lr(dl, dr, disp_checked=out[2])
    for name, o, w in zip(("left", "right", "checked"), out, want):
        np.testing.assert_array_equal(_got(o), w, err_msg=name + " alone")
    r = ct.BlockMatcherCensus()
    r.configure(0, W, H, D, left_to_right=False, disp_min=dmin)
    r.process(out[1], dl, dr)
    np.testing.assert_array_equal(_got(out[1]), want[1])
    assert m.device_status() == 0 and r.device_status() == 0


def test_calls_in_turn_with_the_cuda_core_pass(ct, oracle, cuda):
    """Right-view keys of many calls, of other pairs and of both kinds of pass
    do not reach a later call's maps."""
    W, H, D = 333, 47, 128
    pairs = []
    for seed in (1, 2, 3):
        L, R, _, _ = ct.synth_pair(1 + seed % 2, seed, W, H, D - 1)
        pairs.append((to_dev(L, cuda), to_dev(R, cuda), _want(oracle, L, R, D, 0, torch.int16)))
    a, b = ct.BlockMatcherCensus(), ct.BlockMatcherCensus()
    a.configure(0, W, H, D)
    b.configure(0, W, H, D)
    out = [ct.alloc_image(H, W, torch.int16, cuda) for _ in range(3)]
    for k in range(70):  # more than twice the tags a key has
        if k == 40:  # from here on this handle runs the CUDA-core pass
            b.set_tuning(36, 4)
        m = b if k % 2 else a
        dl, dr, want = pairs[k % 3]
        if k % 7 == 3:
            m.process_lr(dl, dr, disp_rl=out[1])
            np.testing.assert_array_equal(_got(out[1]), want[1], err_msg=str(k))
            continue
        m.process_lr(dl, dr, *out, tol=1)
        if k % 5 == 0 or k > 60:
            for o, w in zip(out, want):
                np.testing.assert_array_equal(_got(o), w, err_msg=str(k))
    assert a.device_status() == 0 and b.device_status() == 0
