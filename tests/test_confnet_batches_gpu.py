"""Gradients of the confidence net on one handle over batches of changing size
(its operand maps are kept per size, its scratch holds what larger batches left)
and from samples at any address. The sums have a fixed order, so every gradient
is bit for bit that of a handle of its own."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _batch(n, seed):
    r = np.random.default_rng(seed)
    x = r.integers(0, 197, (n, 128)).astype(np.uint8)
    x[np.arange(128)[None, :] >= r.integers(60, 200, (n, 1))] = 255
    return x, (r.random(n) < 0.7).astype(np.uint8)


def _grad(ct, cuda, net, xs, ys):
    grad = torch.full((ct.CT_CONFNET_PARAMS,), float("nan"), dtype=torch.float32, device=cuda)
    loss = torch.empty(1, dtype=torch.float32, device=cuda)
    net.loss_grad(xs, ys, grad, loss)
    return grad.cpu().numpy(), loss.item()


def _net(ct, max_batch):
    net = ct.ConfNet()
    net.configure(0, max_batch)
    net.init(5)
    return net


def test_batches_of_changing_size_on_one_handle(ct, cuda):
    shared = _net(ct, 1024)
    for k, n in enumerate((1024, 600, 37, 1, 8, 1023, 37, 256, 1024)):
        x, y = _batch(n, k)
        xs, ys = torch.from_numpy(x).to(cuda), torch.from_numpy(y).to(cuda)
        got, loss = _grad(ct, cuda, shared, xs, ys)
        want, want_loss = _grad(ct, cuda, _net(ct, n), xs, ys)
        np.testing.assert_array_equal(got, want, err_msg=f"{k}: {n} samples")
        assert loss == want_loss and np.isfinite(got).all()
    shared.configure(0, 64)  # other scratch, the size of an earlier batch
    shared.init(5)
    x, y = _batch(37, 99)
    xs, ys = torch.from_numpy(x).to(cuda), torch.from_numpy(y).to(cuda)
    np.testing.assert_array_equal(_grad(ct, cuda, shared, xs, ys)[0], _grad(ct, cuda, _net(ct, 37), xs, ys)[0])
    assert shared.device_status() == 0


@pytest.mark.parametrize("offset", [1, 2, 3])
@pytest.mark.parametrize("n", [1, 37, 300])
def test_samples_at_any_address(ct, cuda, n, offset):
    x, y = _batch(n, n)
    xs, ys = torch.from_numpy(x).to(cuda), torch.from_numpy(y).to(cuda)
    buf = torch.zeros(n * 128 + 8, dtype=torch.uint8, device=cuda)
    odd = buf[offset:offset + n * 128].view(n, 128)
    odd.copy_(xs)
    assert odd.data_ptr() % 4 == offset
    net = _net(ct, n)
    got, want = _grad(ct, cuda, net, odd, ys), _grad(ct, cuda, net, xs, ys)
    np.testing.assert_array_equal(got[0], want[0])
    assert got[1] == want[1]
    a, b = (torch.empty(n, dtype=torch.float32, device=cuda) for _ in range(2))
    net.scores(a, odd)
    net.scores(b, xs)
    np.testing.assert_array_equal(a.cpu().numpy(), b.cpu().numpy())
    assert net.device_status() == 0
