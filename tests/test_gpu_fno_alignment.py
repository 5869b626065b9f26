"""Inputs of the surrogate that start on a 4-byte boundary only.  The tcgen05
products copy their input in 16-byte pieces, so an input off that grid takes
the general product (a network) or is refused (the products' own entries).

Tolerance: the two products may differ by FP32 rounding of the lift, which
moves a later operand by at most one BF16 step (2^-8) where it crosses a
rounding boundary: 1e-3 in norm for the output and every gradient."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("proj,bf16_act", [(32, "0"), (128, "0"), (128, "1")])
def test_network_input_on_any_element(lib, monkeypatch, proj, bf16_act):
    from atmosphericturbulencesimul_gb300 import fno as F
    monkeypatch.setenv("ATMWFS_FNO_BF16_ACT", bf16_act)
    grid = 256 if proj == 128 else 64
    m = F.Surrogate(F.FnoConfig(nin=8, width=64, modes=32 if proj == 128 else 8, layers=1, proj=proj, nout=2, grid=grid), seed=4)
    g = torch.Generator().manual_seed(proj)
    n = 2 * 8 * grid * grid
    buf = torch.randn(n + 4, generator=g).cuda()
    t = torch.randn(2, 2, grid, grid, generator=g).cuda()
    out, grads = [], []
    for off in (0, 1):
        x = torch.empty(n + 4, device="cuda")[off:off + n].view(2, 8, grid, grid)
        x.copy_(buf[:n].view_as(x))
        assert x.data_ptr() % 16 == 4 * off
        out.append(m.forward(x).cpu())
        m.zero_grads()
        m.loss_grad(x, t, out=torch.empty_like(t))
        grads.append(m.get_grads())
    m.close()
    assert ((out[0] - out[1]).norm() / out[0].norm()).item() < 1e-3
    assert np.linalg.norm(grads[0] - grads[1]) / np.linalg.norm(grads[0]) < 1e-3


def test_products_refuse_inputs_off_16_bytes(lib):
    W = torch.zeros(512 * 512, dtype=torch.bfloat16, device="cuda")
    X = torch.zeros(512 * 1024 + 4, device="cuda")
    out = torch.zeros(512 * 1024, device="cuda")
    p = lambda t, off=0: C.c_void_p(t.data_ptr() + 4 * off)
    for o, c in ((64, 64), (128, 64), (64, 8)):
        assert lib.atmwfs_fno_pointwise_dev(p(W), o, c, p(X), p(out), 1, 1024, 0.0, None, None, 1, None) == 0
        assert lib.atmwfs_fno_pointwise_dev(p(W), o, c, p(X, 1), p(out), 1, 1024, 0.0, None, None, 1, None) != 0
    for o, c in ((64, 512), (512, 64)):
        assert lib.atmwfs_fno_spectral_dev(p(W), o, c, p(X), p(out), 1024, 1, None) == 0
        assert lib.atmwfs_fno_spectral_dev(p(W), o, c, p(X, 2), p(out), 1024, 1, None) != 0
    torch.cuda.synchronize()
