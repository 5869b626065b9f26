"""Chromatic PSFs at the sizes whose row and column passes have a shape of their
own, against the FP64 oracle: fewer steps than the column pass has lanes and
more, one step, and (2048) rows above 48 KB of shared memory.

Tolerance: FP32 transforms against FP64, relative max error 2e-5 of the image
maximum (the bar of the other PSF tests)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,steps,apo", [(64, 17, 0.3), (256, 3, 0.0), (256, 18, 0.3), (512, 5, 0.0), (1024, 4, 0.3), (2048, 3, 1.0)])
def test_chromatic_psf_sizes(lib, oracle64, n, steps, apo):
    from atmosphericturbulencesimul_gb300 import psf as P
    y, x = np.mgrid[0:n, 0:n] - (n / 2 - 0.5)
    amp = (np.hypot(x, y) < n / 4).astype(np.float32)
    pha = (np.sin(x / 17.0) * np.cos(y / 23.0) * 2.0 * amp).astype(np.float32)
    got = P.chromat_psf(amp, pha, 0.7, 1.4, steps, apo)
    ref = oracle64.chromat_psf(amp, pha, 0.7, 1.4, steps, apo)
    assert ref.max() > 0
    assert np.abs(got - ref).max() / ref.max() < 2e-5
