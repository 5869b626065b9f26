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


def test_workspaces_of_concurrent_and_captured_calls(lib):
    """The calls' device workspaces come from one pool: transforms of several
    sizes issued by two host threads on streams of their own give the results
    of calls made one by one, and a captured call can be replayed."""
    import threading

    import torch
    from atmosphericturbulencesimul_gb300 import _lib

    def call(a, out, st):
        _lib.check(lib.atmwfs_fft2d_dev(C.c_void_p(a.data_ptr()), C.c_void_p(out.data_ptr()), a.shape[0], -1, C.c_void_p(st)))

    sizes = [64, 4096, 512, 256, 4096, 1024]
    g = torch.Generator(device="cuda").manual_seed(5)
    ins = [torch.randn((n, n), dtype=torch.complex64, device="cuda", generator=g) for n in sizes]
    want = [torch.empty_like(a) for a in ins]
    for a, o in zip(ins, want):
        call(a, o, 0)
    torch.cuda.synchronize()
    outs = [[torch.zeros_like(a) for a in ins] for _ in range(2)]

    def work(k):
        st = torch.cuda.Stream()
        for _ in range(5):
            for a, o in zip(ins, outs[k]):
                call(a, o, st.cuda_stream)
        st.synchronize()

    ts = [threading.Thread(target=work, args=(k,)) for k in range(2)]
    [t.start() for t in ts]
    [t.join() for t in ts]
    for k in range(2):
        assert all(torch.equal(o, w) for o, w in zip(outs[k], want))
    graph, out = torch.cuda.CUDAGraph(), torch.zeros_like(ins[2])
    with torch.cuda.graph(graph):
        call(ins[2], out, torch.cuda.current_stream().cuda_stream)
    out.zero_()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, want[2])
