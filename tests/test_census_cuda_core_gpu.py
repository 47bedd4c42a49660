"""The census matcher's CUDA-core pass of both views, which runs by default for
few disparities on large images: against the oracle through that default route,
and on small and degenerate shapes, which run on the tensor cores by default,
with the kernel selected."""
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


def _check(m, dl, dr, want, out):
    for o in out:
        o.fill_(0x2B)
    m.process_lr(dl, dr, *out, tol=1)
    for o, w, name in zip(out, want, ("left", "right", "checked")):
        got = o.cpu().numpy()
        np.testing.assert_array_equal(got.view(w.dtype), w, err_msg=name)


@pytest.mark.parametrize("W,H,D,dmin,dtype", [
    (1280, 720, 32, 3, torch.int16),
    (1023, 601, 47, 0, torch.uint8),
    (801, 603, 1, 7, torch.int16),
])
def test_default_route_of_large_images_with_few_disparities(ct, oracle, cuda, W, H, D, dmin, dtype):
    L, R, _, _ = ct.synth_pair(2, W + D, W, H, D - 1 + dmin)
    m = ct.BlockMatcherCensus()
    m.configure(0, W, H, D, disp_min=dmin)
    assert m.tuning()["strip_height"] < ct.CT_TUNING_TC_LEFT  # no pass on the tensor cores
    _check(m, to_dev(L, cuda), to_dev(R, cuda), _want(oracle, L, R, D, dmin, dtype),
           [ct.alloc_image(H, W, dtype, cuda) for _ in range(3)])
    assert m.device_status() == 0


@pytest.mark.parametrize("W,H,D,dmin,dtype", [
    (8, 8, 1, 0, torch.int16),        # smallest image, one disparity
    (16, 9, 3, 1, torch.int16),       # odd minimum disparity, D tiny
    (96, 64, 1, 0, torch.uint8),      # D = 1
    (67, 43, 40, 0, torch.int16),     # one column tile, D below one disparity block
    (130, 37, 64, 0, torch.int16),    # exactly one block of disparities, two column tiles
    (124, 40, 65, 0, torch.uint8),    # one column tile, D one past a block
    (333, 111, 128, 5, torch.int16),  # odd minimum disparity (relative d = 0 excluded)
    (515, 97, 200, 2, torch.uint8),   # ragged D and width, U8 maps
    (640, 50, 256, 0, torch.int16),
    (60, 30, 20, 50, torch.int16),    # minimum disparity close to the width: most pixels search nothing
    (50, 20, 10, 60, torch.int16),    # minimum disparity beyond the width: no disparity anywhere
])
@pytest.mark.parametrize("dpw", [4, 8])
def test_selected_kernel_is_bit_exact(ct, oracle, cuda, W, H, D, dmin, dtype, dpw):
    L, R, _, _ = ct.synth_pair(1, 700 + W + D, W, H, max(1, dmin + D - 1))
    m = ct.BlockMatcherCensus()
    m.configure(0, W, H, D, disp_min=dmin)
    m.set_tuning(36, dpw)
    _check(m, to_dev(L, cuda), to_dev(R, cuda), _want(oracle, L, R, D, dmin, dtype),
           [ct.alloc_image(H, W, dtype, cuda) for _ in range(3)])
    assert m.device_status() == 0


@pytest.mark.parametrize("dtype", [torch.uint8, torch.int16])
def test_keys_of_many_calls(ct, oracle, cuda, dtype):
    """The right view's keys stay between calls and are told apart by a tag that
    counts down: over more than two rounds of tags, on pairs of different
    disparities, no call meets an earlier one's."""
    W, H, D = 200, 40, 64
    scenes = []
    for kind, seed, dmax in ((1, 31, D - 1), (2, 32, 20), (1, 33, 40)):
        L, R, _, _ = ct.synth_pair(kind, seed, W, H, dmax)
        scenes.append((to_dev(L, cuda), to_dev(R, cuda), _want(oracle, L, R, D, 0, dtype)))
    m = ct.BlockMatcherCensus()
    m.configure(0, W, H, D)
    m.set_tuning(36, 4)
    out = [ct.alloc_image(H, W, dtype, cuda) for _ in range(3)]
    for k in range(70):
        _check(m, *scenes[k % 3], out)
    assert m.device_status() == 0
