"""A batch whose activations do not fit the device is refused, and leaves the
model fit for the batches that do: the activations of the earlier batch are gone
by then, so the next call makes its own.  (The first buffer of the refused batch
alone exceeds the device's memory: nothing is held when it fails.)"""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("width,proj", [(64, 128), (32, 32)])
def test_refused_batch_leaves_the_model_usable(lib, width, proj):
    from atmosphericturbulencesimul_gb300 import fno as F
    m = F.Surrogate(F.FnoConfig(nin=8, width=width, modes=32, layers=1, proj=proj, nout=2, grid=256), seed=2)
    x = torch.randn(2, 8, 256, 256, generator=torch.Generator().manual_seed(1)).cuda()
    want = m.forward(x)
    out = torch.empty_like(want)
    p = lambda t: C.c_void_p(t.data_ptr())
    assert lib.atmwfs_fno_forward(m._h, p(x), p(out), 200000, None) == 2   # ATMWFS_ERR_NOMEM
    assert torch.equal(m.forward(x), want)
    assert m.loss_grad(x, torch.zeros_like(want)) > 0
    m.close()
