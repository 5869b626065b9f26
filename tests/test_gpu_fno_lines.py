"""The x transforms that leave with the activations: lines (sample, row) are
dealt to persistent CTAs, each of which stores a line's spectrum one line
later.  A sample's output does not depend on how many lines there are (fewer
than the CTAs, one more round, several), and the lift with its transform (8
input planes) gives what the separate lift and transform give (5 planes, the
other three weighted 0).

Tolerances: the same kernels on the same values give the same bits; the two
lifts may differ by FP32 rounding, which moves a product operand by at most one
BF16 step (2^-8) where it crosses a rounding boundary: 1e-3 in norm."""
import numpy as np
import pytest

from oracle import fno_oracle as fo

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def net(nin, layers, p):
    from atmosphericturbulencesimul_gb300 import fno as F
    cfg = fo.Cfg(nin=nin, width=64, modes=32, layers=layers, proj=128, nout=2, grid=256)
    m = F.Surrogate(F.FnoConfig(**cfg.__dict__), seed=1)
    m.set_params(p.astype(np.float32))
    return m


@pytest.mark.parametrize("layers,batch", [(1, 2), (2, 2), (3, 5)])
def test_lines_and_lifts(lib, layers, batch):
    cfg8 = fo.Cfg(nin=8, width=64, modes=32, layers=layers, proj=128, nout=2, grid=256)
    p8 = fo.init_params(cfg8, 7)
    o, n = fo.layout(cfg8)["lift_W"]
    w = p8[o:o + n].reshape(64, 8)
    w[:, 5:] = 0.0
    p8[o:o + n] = w.ravel()
    p5 = np.concatenate([p8[:o], w[:, :5].ravel(), p8[o + n:]])
    x = torch.randn(batch, 8, 256, 256, generator=torch.Generator().manual_seed(layers)).cuda()
    m8, m5 = net(8, layers, p8), net(5, layers, p5)
    whole = m8.forward(x)
    for b in range(batch):
        assert torch.equal(whole[b:b + 1], m8.forward(x[b:b + 1].contiguous()))
    other = m5.forward(x[:, :5].contiguous())
    assert ((whole - other).norm() / other.norm()).item() < 1e-3
    assert lib.atmwfs_fno_umma_status(0) == 0
    m8.close()
    m5.close()
