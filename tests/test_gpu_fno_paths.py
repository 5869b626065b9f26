"""The fused kernels of the default shape against the separate products (every
product on mma.sync, ATMWFS_FNO_UMMA=0, in a process of its own since the
switch is read once), element by element: the output and every gradient tensor
in the maximum norm, so that an error confined to a few pixels, an edge column
or one mode shows.

Tolerance: both round the same operands to BF16; the sums in between are added
in another FP32 order, which moves an operand by one BF16 step (2^-8) where it
crosses a rounding boundary.  Eight such steps among the 128 terms of an output,
each 2^-8 of a term of four times the terms' rms, are 4e-3 of a maximum of three
times the output's rms: 5e-3 of a tensor's largest element."""
import os
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

from oracle import fno_oracle as fo

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

ROOT = Path(__file__).resolve().parent.parent


def run(layers, batch, nin):
    from atmosphericturbulencesimul_gb300 import fno as F
    cfg = fo.Cfg(nin=nin, width=64, modes=32, layers=layers, proj=128, nout=2, grid=256)
    p = fo.init_params(cfg, 3)
    for name, (o, n) in fo.layout(cfg).items():
        if name.startswith("R"):
            p[o:o + n] *= 30.0          # spectral weights that carry part of the output
    g = torch.Generator().manual_seed(batch)
    x = torch.randn(batch, nin, 256, 256, generator=g).cuda()
    t = (torch.randn(batch, 2, 256, 256, generator=g) * 0.3).cuda()
    m = F.Surrogate(F.FnoConfig(**cfg.__dict__), seed=1)
    m.set_params(p.astype(np.float32))
    out = torch.empty_like(t)
    m.zero_grads()
    m.loss_grad(x, t, out=out)
    g = m.get_grads()
    m.close()
    return out.cpu().numpy(), g, fo.layout(cfg)


@pytest.mark.parametrize("layers,batch,nin", [(1, 2, 8), (2, 3, 8), (2, 1, 5)])
def test_fused_and_separate_products_agree(lib, tmp_path, layers, batch, nin):
    code = ("import sys; sys.path[:0] = [%r, %r]\nimport numpy as np, test_gpu_fno_paths as t\n"
            "o, g, _ = t.run(%d, %d, %d)\nnp.savez(%r, o=o, g=g)\n") % (
                str(ROOT), str(ROOT / "tests"), layers, batch, nin, str(tmp_path / "sep.npz"))
    subprocess.run([sys.executable, "-c", code], check=True, env={**os.environ, "ATMWFS_FNO_UMMA": "0"}, timeout=300)
    sep = np.load(tmp_path / "sep.npz")
    out, grads, lay = run(layers, batch, nin)
    assert np.abs(out - sep["o"]).max() < 5e-3 * np.abs(sep["o"]).max()
    for name, (o, n) in lay.items():
        if name == "_total":
            continue
        a, b = grads[o:o + n], sep["g"][o:o + n]
        assert np.abs(a - b).max() < 5e-3 * np.abs(b).max(), (name, np.abs(a - b).max() / np.abs(b).max())
