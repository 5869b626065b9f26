"""The surrogate's fused kernels (the default shape: grid 256, 32 modes, width
64, projection 128) against the FP64 oracle: inference, loss and every
parameter gradient, for one layer (no activation between the x transforms) and
two, with a batch whose lines are fewer than the persistent kernels' CTAs (1),
odd and beyond one sample block of the mode mixing (3, 9), and accumulation of
gradients over two calls.

Tolerances: every product operand is rounded to BF16 (relative 2e-2 in norm per
tensor, as the other surrogate tests); inference and the training forward give
the same bits."""
import numpy as np
import pytest

from oracle import fno_oracle as fo

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("layers,batch", [(1, 1), (2, 3), (1, 9)])
def test_fused_shape_matches_oracle(lib, layers, batch):
    from atmosphericturbulencesimul_gb300 import fno as F
    cfg = fo.Cfg(nin=8, width=64, modes=32, layers=layers, proj=128, nout=2, grid=256)
    rng = np.random.default_rng(layers * 10 + batch)
    p = fo.init_params(cfg, 3)
    lay = fo.layout(cfg)
    for name, (o, n) in lay.items():
        if name.startswith("R"):
            p[o:o + n] *= 30.0          # spectral weights that carry part of the output
    x = rng.standard_normal((batch, cfg.nin, cfg.grid, cfg.grid)).astype(np.float32)
    t = (rng.standard_normal((batch, cfg.nout, cfg.grid, cfg.grid)) * 0.3).astype(np.float32)
    m = F.Surrogate(F.FnoConfig(**cfg.__dict__), seed=1)
    m.set_params(p.astype(np.float32))
    xt, tt = torch.tensor(x, device="cuda"), torch.tensor(t, device="cuda")
    inf = m.forward(xt)
    out = torch.empty_like(inf)
    m.zero_grads()
    loss = m.loss_grad(xt, tt, out=out)
    torch.cuda.synchronize()
    assert torch.equal(inf, out)
    g = m.get_grads()
    lo, go = fo.loss_grad(p, x, t, cfg)
    ref = fo.forward(p, x, cfg)
    assert np.linalg.norm(out.cpu().numpy() - ref) / np.linalg.norm(ref) < 2e-2
    assert abs(loss - lo) / lo < 1e-2
    for name, (o, n) in lay.items():
        if name == "_total":
            continue
        err = np.linalg.norm(g[o:o + n] - go[o:o + n]) / np.linalg.norm(go[o:o + n])
        assert err < 2e-2, (name, err)
    m.loss_grad(xt, tt, out=out)        # gradients accumulate
    g2 = m.get_grads()
    assert np.linalg.norm(g2 - 2 * g) / np.linalg.norm(g) < 1e-4
    assert lib.atmwfs_fno_umma_status(0) == 0
    m.close()
