"""The surrogate's work area must lie on a 16-byte boundary: one that does not is refused before any launch,
and the network goes on working."""

import ctypes as C

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("off", [2, 4, 8])
def test_work_off_its_boundary_is_refused(off):
    from epsr_python_translation_b200.surrogate import IN, SurrogateNet, _p, _stream
    net = SurrogateNet(seed=3)
    x = torch.randn(128, IN, device="cuda").to(torch.bfloat16)
    want = net.forward(x)
    y = torch.full((128,), 7.0, device="cuda")
    nb = int(net.lib.epsr_mlp_work_bytes(128))
    work = torch.zeros(nb + 256, dtype=torch.uint8, device="cuda")
    at = C.c_void_p(work.data_ptr() + off)
    p0 = net.params()
    t = torch.zeros(64, device="cuda")
    assert net.lib.epsr_mlp_forward(C.byref(net.c), _p(x), 128, _p(y), at, nb, _stream()) == 1
    assert net.lib.epsr_mlp_train_step(C.byref(net.c), _p(x), _p(x.t().contiguous()), 128, 0, 128, _p(t), 1e-3, 1, None,
                                       at, nb, _stream()) == 1
    torch.cuda.synchronize()
    assert torch.all(y == 7.0) and not work.any()
    assert all((p0[k] == v).all() for k, v in net.params().items())
    assert torch.equal(net.forward(x), want)
