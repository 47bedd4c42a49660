"""Waits of the tensor-core census pass that give up, without a GPU fault: with
a limit of no or very few polls the warps' waits run out while the MMAs are on
their way. The call ends, reports CT_ETIMEOUT, writes nothing outside its maps,
and later calls are right again."""
import numpy as np
import pytest
import torch

from conftest import to_dev

pytestmark = pytest.mark.gpu

NORMAL = 65536


def _guarded(ct, cuda, H, W):
    """A U16 map between guard rows, and the allocation."""
    whole = ct.alloc_image(H + 4, W, torch.int16, cuda)
    whole.fill_(0x2B2B)
    return whole[2:H + 2], whole


def _guards_intact(whole):
    a = whole.cpu().numpy()
    assert (a[:2] == 0x2B2B).all() and (a[-2:] == 0x2B2B).all()


@pytest.mark.parametrize("W,H,D", [
    (339, 37, 128),   # a last pair with one tile
    (300, 90, 200),   # tiles that share their left pixels
    (8, 8, 48),
])
def test_matcher_waits_that_give_up(ct, oracle, cuda, W, H, D):
    L, R, _, _ = ct.synth_pair(1, 900 + W, W, H, D - 1)
    dl, dr = to_dev(L, cuda), to_dev(R, cuda)
    lr, _ = oracle.match_census(L, R, D, 2, True)
    rl, _ = oracle.match_census(L, R, D, 2, False)
    a, b = oracle.to_u16(lr), oracle.to_u16(rl)
    want = a, b, oracle.crosscheck_codes(a, b, 1, True, frame=False)[0]
    m = ct.BlockMatcherCensus()
    m.configure(0, W, H, D)
    maps = [_guarded(ct, cuda, H, W) for _ in range(3)]

    def call():
        m.process_lr(dl, dr, *(v for v, _ in maps), tol=1)
        status = m.device_status()
        for _, whole in maps:
            _guards_intact(whole)
        return status

    for polls in (0, 1, 0, 2):
        m.test_wait_limit(polls)
        status = call()
        assert status == ct.CT_ETIMEOUT or (polls and status == 0)
    m.test_wait_limit(NORMAL)
    for _ in range(2):
        assert call() == 0
        for (v, _), w in zip(maps, want):
            np.testing.assert_array_equal(v.cpu().numpy().view(np.uint16), w)


def test_batch_waits_that_give_up(ct, cuda):
    shapes = [(320, 240, 64), (257, 100, 200), (640, 120, 128)]
    pairs, whole = [], []
    for i, (W, H, D) in enumerate(shapes):
        L, R, _, _ = ct.synth_pair(1, 40 + i, W, H, D - 1)
        v, g = _guarded(ct, cuda, H, W)
        pairs.append((to_dev(L, cuda), to_dev(R, cuda), v))
        whole.append(g)
    m = ct.BatchStereo()
    m.configure(0, shapes, tol=1)
    m.process(pairs)
    assert m.device_status() == 0
    want = [p[2].cpu().numpy() for p in pairs]
    m.test_wait_limit(0)
    m.process(pairs)
    assert m.device_status() == ct.CT_ETIMEOUT
    m.test_wait_limit(NORMAL)
    m.configure(0, shapes, tol=1)
    m.process(pairs)
    assert m.device_status() == 0
    for p, g, w in zip(pairs, whole, want):
        _guards_intact(g)
        np.testing.assert_array_equal(p[2].cpu().numpy(), w)


def test_wait_limit_checks_its_arguments(ct, cuda):
    m = ct.BlockMatcherCensus()
    with pytest.raises(ct.CtError) as e:
        m.test_wait_limit(NORMAL + 1)
    assert e.value.code == ct.CT_EINVAL
    with pytest.raises(ct.CtError) as e:
        ct.BlockMatcherNCC().test_wait_limit(1)
    assert e.value.code == ct.CT_ESTATE
