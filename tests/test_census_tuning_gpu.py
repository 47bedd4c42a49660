"""The census matcher's tuning, saved and set on another handle, carries which
kernel runs each kind of pass. The tensor-core pass shows itself by its waits:
with a limit of no polls its calls report CT_ETIMEOUT."""
import numpy as np
import pytest
import torch

from conftest import to_dev

pytestmark = pytest.mark.gpu


def _on_tensor_cores(ct, cuda, m, dl, dr):
    """Which kinds of pass of the handle run on the tensor cores."""
    H, W = dl.shape
    out = ct.alloc_image(H, W, torch.int16, cuda)
    m.test_wait_limit(0)
    kinds = {}
    for name, maps in (("left", {"disp_lr": out}), ("right", {"disp_rl": out}), ("checked", {"disp_checked": out})):
        m.process_lr(dl, dr, **maps)
        kinds[name] = m.device_status() == ct.CT_ETIMEOUT
    m.test_wait_limit(65536)
    return kinds


@pytest.mark.parametrize("W,H,D", [
    (333, 47, 128),    # every pass on the tensor cores by default
    (333, 47, 64),     # all but the right view alone
    (1280, 720, 32),   # none
])
@pytest.mark.parametrize("tune", [False, True])
def test_saved_tuning_runs_the_same_kernels(ct, oracle, cuda, W, H, D, tune):
    L, R, _, _ = ct.synth_pair(1, 60 + D, W, H, D - 1)
    dl, dr = to_dev(L, cuda), to_dev(R, cuda)
    a, b = ct.BlockMatcherCensus(), ct.BlockMatcherCensus()
    for m in (a, b):
        m.configure(0, W, H, D)
    saved = a.autotune(dl, dr) if tune else a.tuning()
    b.set_tuning(36, 4)
    assert not any(_on_tensor_cores(ct, cuda, b, dl, dr).values())
    b.set_tuning(**saved)
    assert b.tuning() == saved
    kinds = _on_tensor_cores(ct, cuda, a, dl, dr)
    assert _on_tensor_cores(ct, cuda, b, dl, dr) == kinds
    if not tune:
        assert kinds == {"left": D >= 48, "right": D > 64, "checked": D >= 48}
    out = ct.alloc_image(H, W, torch.int16, cuda)
    b.process(out, dl, dr)
    np.testing.assert_array_equal(out.cpu().numpy().view(np.uint16), oracle.to_u16(oracle.match_census(L, R, D)[0]))
    assert a.device_status() == 0 and b.device_status() == 0


def test_each_kind_of_pass_has_a_kernel_of_its_own(ct, oracle, cuda):
    """(The autotuner times the pass of both views by itself: which kernel is the
    faster one for the left view alone does not decide it.)"""
    W, H, D = 333, 47, 100
    L, R, _, _ = ct.synth_pair(2, 5, W, H, D - 1)
    dl, dr = to_dev(L, cuda), to_dev(R, cuda)
    lr, rl = (oracle.to_u16(oracle.match_census(L, R, D, 2, left)[0]) for left in (True, False))
    want = lr, rl, oracle.crosscheck_codes(lr, rl, 1, True, frame=False)[0]
    m = ct.BlockMatcherCensus()
    m.configure(0, W, H, D)
    out = [ct.alloc_image(H, W, torch.int16, cuda) for _ in range(3)]
    for k in range(8):
        m.set_tuning(36 + k * ct.CT_TUNING_TC_LEFT, 4)
        assert _on_tensor_cores(ct, cuda, m, dl, dr) == {"left": bool(k & 1), "right": bool(k & 2),
                                                         "checked": bool(k & 4)}
        m.process_lr(dl, dr, disp_lr=out[0])
        m.process_lr(dl, dr, disp_rl=out[1])
        m.process_lr(dl, dr, disp_checked=out[2])
        for o, w in zip(out, want):
            np.testing.assert_array_equal(o.cpu().numpy().view(np.uint16), w)
    assert m.device_status() == 0


def test_tunings_of_no_kernel_are_refused(ct, cuda):
    m = ct.BlockMatcherCensus()
    m.configure(0, 160, 96, 64)
    before = m.tuning()
    for th, dpw in ((12, 4), (516, 4), (ct.CT_TUNING_TC_LEFT, 4), (ct.CT_TUNING_TC_LEFT + 12, 4), (-4, 4),
                    (36 - ct.CT_TUNING_TC_LEFT, 4), (4 * ct.CT_TUNING_TC_LEFT * 8 + 36, 4), (ct.CT_TUNING_TC_LEFT + 36, 5)):
        with pytest.raises(ct.CtError) as e:
            m.set_tuning(th, dpw)
        assert e.value.code == ct.CT_EINVAL
    assert m.tuning() == before
