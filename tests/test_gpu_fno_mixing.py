"""The mode mixing outside the fused shape, on both sides of its rule: one
thread per output value (widths of 20 and 96) and blocks of eight samples where
the weights leave room for one CTA of the first (width 128, and width 64 with
many samples), with batches below, above and a multiple of eight.  Forward and
every gradient against the FP64 oracle, with spectral weights that carry most
of the output.

Tolerance: every product operand is rounded to BF16 (relative 2e-2 in norm per
tensor, as the other surrogate tests)."""
import numpy as np
import pytest

from oracle import fno_oracle as fo

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


@pytest.mark.parametrize("width,batch", [(20, 1), (20, 9), (96, 3), (128, 1), (128, 9), (64, 160)])
def test_mode_mixing_matches_oracle(lib, width, batch):
    from atmosphericturbulencesimul_gb300 import fno as F
    cfg = fo.Cfg(nin=3, width=width, modes=4, layers=1, proj=16, nout=2, grid=16)
    rng = np.random.default_rng(width + batch)
    p = fo.init_params(cfg, 5)
    lay = fo.layout(cfg)
    o, n = lay["R0"]
    p[o:o + n] *= 30.0
    x = rng.standard_normal((batch, cfg.nin, cfg.grid, cfg.grid)).astype(np.float32)
    t = (rng.standard_normal((batch, cfg.nout, cfg.grid, cfg.grid)) * 0.3).astype(np.float32)
    m = F.Surrogate(F.FnoConfig(**cfg.__dict__), seed=1)
    m.set_params(p.astype(np.float32))
    out = torch.empty(batch, cfg.nout, cfg.grid, cfg.grid, device="cuda")
    m.zero_grads()
    m.loss_grad(torch.tensor(x, device="cuda"), torch.tensor(t, device="cuda"), out=out)
    g = m.get_grads()
    m.close()
    ref = fo.forward(p, x, cfg)
    assert np.linalg.norm(out.cpu().numpy() - ref) / np.linalg.norm(ref) < 2e-2
    _, go = fo.loss_grad(p, x, t, cfg)
    for name, (o, n) in lay.items():
        if name != "_total":
            err = np.linalg.norm(g[o:o + n] - go[o:o + n]) / np.linalg.norm(go[o:o + n])
            assert err < 2e-2, (name, err)
