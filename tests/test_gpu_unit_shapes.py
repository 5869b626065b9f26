"""The device transforms through the C ABI at every size their launch shapes
differ at, against numpy in double: row counts per CTA by size up to 2048, the
clusters of eight rows above, both directions, in place, and buffers aligned
to one complex value only.

Tolerance: FP32 butterflies against FP64, log2(n^2) <= 26 levels of at most a
few roundings of 6e-8 each: relative max error <= 2e-5 (the bar of the other
transform tests)."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
TOL = 2e-5


def _run(lib, a, sign, off_in, off_out, in_place):
    import torch
    from atmosphericturbulencesimul_gb300 import _lib
    n = a.shape[0]
    buf = torch.empty(n * n + 2, dtype=torch.complex64, device="cuda")
    out = torch.full((n * n + 2,), 7.0, dtype=torch.complex64, device="cuda")
    src = buf[off_in:off_in + n * n]
    src.copy_(torch.from_numpy(a.reshape(-1)))
    dst = src if in_place else out[off_out:off_out + n * n]
    _lib.check(lib.atmwfs_fft2d_dev(C.c_void_p(src.data_ptr()), C.c_void_p(dst.data_ptr()), n, sign, None))
    torch.cuda.synchronize()
    if not in_place:  # nothing outside the image is written
        assert (out[:off_out] == 7).all() and (out[off_out + n * n:] == 7).all()
    return dst.cpu().numpy().reshape(n, n)


@pytest.mark.parametrize("n,sign,off_in,off_out,in_place", [
    (64, -1, 0, 0, False), (128, 1, 0, 0, False), (256, -1, 1, 1, False), (512, 1, 0, 0, True),
    (1024, -1, 0, 1, False), (2048, 1, 0, 0, False), (4096, -1, 0, 1, False), (4096, 1, 1, 0, False),
    (4096, -1, 0, 0, True), (8192, 1, 0, 1, False),
])
def test_fft2d_dev_launch_shapes(lib, n, sign, off_in, off_out, in_place):
    rng = np.random.default_rng(n + sign)
    a = (rng.standard_normal((n, n), np.float32) + 1j * rng.standard_normal((n, n), np.float32)).astype(np.complex64)
    got = _run(lib, a, sign, off_in, off_out, in_place)
    ref = np.fft.fft2(a.astype(np.complex128)) if sign < 0 else np.fft.ifft2(a.astype(np.complex128)) * n * n
    assert np.abs(got - ref).max() / np.abs(ref).max() < TOL
