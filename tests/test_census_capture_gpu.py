"""Census matcher calls captured into a CUDA graph and replayed between direct
calls of the same handle: every map is that call's own."""
import numpy as np
import pytest
import torch

from conftest import to_dev

pytestmark = pytest.mark.gpu

W, H, D = 333, 47, 128


def _want(oracle, L, R):
    lr, _ = oracle.match_census(L, R, D, 2, True)
    rl, _ = oracle.match_census(L, R, D, 2, False)
    a, b = oracle.to_u16(lr), oracle.to_u16(rl)
    return a, b, oracle.crosscheck_codes(a, b, 1, True, frame=False)[0]


@pytest.fixture
def scenes(ct, oracle, cuda):
    """Three pairs with their maps, and the image buffers that calls read."""
    out = []
    for seed in (1, 2, 3):
        L, R, _, _ = ct.synth_pair(1 + seed % 2, 70 + seed, W, H, D - 1)
        out.append((to_dev(L, cuda), to_dev(R, cuda), _want(oracle, L, R)))
    return out, to_dev(np.zeros((H, W), np.uint8), cuda), to_dev(np.zeros((H, W), np.uint8), cuda)


def _maps(ct, cuda):
    return [ct.alloc_image(H, W, torch.int16, cuda) for _ in range(3)]


def _capture(f):
    g = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(g):
        f()
    return g


def _same(got, want, msg):
    np.testing.assert_array_equal(got.cpu().numpy().view(np.uint16), want, err_msg=msg)


@pytest.mark.parametrize("cuda_cores", [False, True])  # the kernel of the direct calls
def test_right_view_replays_between_direct_calls(ct, cuda, scenes, cuda_cores):
    scenes, left, right = scenes
    m = ct.BlockMatcherCensus()
    m.configure(0, W, H, D)
    alone, out = _maps(ct, cuda)[0], _maps(ct, cuda)
    m.process_lr(left, right, disp_rl=alone)
    g = _capture(lambda: m.process_lr(left, right, disp_rl=alone))  # on the tensor cores
    if cuda_cores:
        m.set_tuning(36, 4)
    for k in range(40):
        dl, dr, want = scenes[k % 3]
        m.process_lr(dl, dr, *out, tol=1)
        for o, w, name in zip(out, want, ("left", "right", "checked")):
            _same(o, w, f"call {k} {name}")
        if k % 4 == 2:
            dl, dr, want = scenes[(k + 1) % 3]
            left.copy_(dl)
            right.copy_(dr)
            g.replay()
            _same(alone, want[1], f"replay {k}")
    assert m.device_status() == 0


@pytest.mark.parametrize("cuda_cores", [False, True])
def test_checked_replays_between_direct_calls(ct, cuda, scenes, cuda_cores):
    """Every replay's keys are its own: neither an earlier replay's, with the
    same tag, nor those of the direct calls between."""
    scenes, left, right = scenes
    m = ct.BlockMatcherCensus()
    m.configure(0, W, H, D)
    if cuda_cores:
        m.set_tuning(36, 4)
    out, direct = _maps(ct, cuda), _maps(ct, cuda)
    m.process_lr(left, right, *out, tol=1)
    g = _capture(lambda: m.process_lr(left, right, *out, tol=1))
    for k in range(40):
        dl, dr, want = scenes[k % 3]
        left.copy_(dl)
        right.copy_(dr)
        g.replay()
        for o, w, name in zip(out, want, ("left", "right", "checked")):
            _same(o, w, f"replay {k} {name}")
        if k % 2:
            dl, dr, want = scenes[(k + 1) % 3]
            m.process_lr(dl, dr, *direct, tol=1)
            for o, w, name in zip(direct, want, ("left", "right", "checked")):
                _same(o, w, f"call {k} {name}")
    assert m.device_status() == 0
