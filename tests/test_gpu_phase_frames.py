"""Phase-only frames (WAVEFRONT_AMPLITUDE 0) against the FP64 oracle's
geometric phase sum (AtmosphericTurbulence.c:2909-2916) at the edges of their
kernel: every grid size (rows and columns per CTA differ), crops off the row
tiles, one layer (one tile buffer), two and sixteen (both buffers reused),
Scoeff equal on all layers (one job per direction) and layer dependent (one
job per instance), and one direction holding several grids and crops.

Tolerances: the bars of the series parity tests (series_case.compare)."""
import numpy as np
import pytest

from series_case import Case, compare

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,Wout,L,flat", [
    (64, 64, 1, True), (64, 37, 2, False), (128, 100, 16, True), (256, 255, 3, False), (512, 401, 2, True),
    (1024, 1021, 4, False), (2048, 1803, 3, True),
])
def test_phase_only_frames(lib, oracle64, W, Wout, L, flat):
    rng = np.random.default_rng(W + L)
    case = Case(alt=[500.0 * k for k in range(L)], cn2=list(rng.uniform(0.1, 1.0, L)), speed=list(rng.uniform(5, 30, L)),
                direction=list(rng.uniform(0, 6.28, L)), M=512, W=W, Wout=Wout, amplitude=0, flat_scoeff=flat,
                sci=[(1.6e-6, 0.0, 0.0), (0.8e-6, 2e-5, -1e-5), (2.2e-6, 2e-5, -1e-5, max(64, W // 2), max(64, W // 2) - 3)])
    ms = compare(case, oracle64, 2)
    assert len(ms) == 2 * 4
