"""The surrogate's forward pass where its tiles end: a row's value depends on that row alone, so any number
of rows gives the same bits as the whole batch; and parameters off a 16-byte boundary (read one by one) give
the same bits as aligned ones.  One training step of 128 and of 384 rows does what three steps' sums say:
the loss is the sum over its 128-row parts to float32 rounding (2^-20 of the sum, 64 pairs a part)."""

import ctypes as C

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _net(seed=3):
    from epsr_python_translation_b200.surrogate import H, IN, SurrogateNet
    rng = np.random.default_rng(seed)
    r = lambda *s: rng.standard_normal(s)  # noqa: E731
    return SurrogateNet(params=dict(w1=r(H, IN) / 36, b1=0.1 * r(H), w2=r(H, H) / 11, b2=0.1 * r(H), w3=r(H) / 11,
                                    b3=0.1 * r(1)))


def _x(rows):
    g = torch.Generator().manual_seed(5)
    return torch.randint(0, 5, (rows, 1280), generator=g).to(torch.bfloat16).cuda()


@pytest.mark.parametrize("rows", [1, 31, 33, 127, 128, 129, 300])
def test_rows_are_independent(rows):
    net, x = _net(), _x(512)
    y = net.forward(x).cpu()
    assert torch.isfinite(y).all() and y.std() > 0
    part = net.forward(x[512 - rows:].contiguous()).cpu()
    net.check_status()
    assert torch.equal(part, y[512 - rows:])


def test_unaligned_parameters():
    net, x = _net(), _x(200)
    y = net.forward(x).cpu()
    keep = []
    for k in ("b1", "b2", "w3"):
        t = torch.zeros(129, device="cuda")
        t[1:] = getattr(net, k)
        keep.append(t)
        setattr(net.c, k, C.c_void_p(t.data_ptr() + 4))
    assert torch.equal(net.forward(x).cpu(), y)
    net.check_status()


@pytest.mark.parametrize("rows", [128, 384])
def test_loss_is_the_sum_of_its_parts(rows):
    x = _x(rows)
    xt = x.t().contiguous()
    t = torch.linspace(-1, 1, rows // 2, device="cuda")
    loss = torch.zeros(1, device="cuda")
    net = _net()
    net.train_step(x, xt, 0, rows, t, 0.0, loss=loss)
    total = 0.0
    for r0 in range(0, rows, 128):
        part = torch.zeros(1, device="cuda")
        other = _net()
        other.train_step(x, xt, r0, 128, t, 0.0, loss=part)
        total += float(part)
    y = _net().forward(x).double().cpu()
    s = 0.5 * (y[0::2] - y[1::2])
    ref = float(((s - t.double().cpu()) ** 2).sum())
    assert abs(float(loss) - total) <= 2.0 ** -20 * total
    assert abs(float(loss) - ref) <= 2.0 ** -18 * ref
