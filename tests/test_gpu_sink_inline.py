"""Sinks of a context with one ring slot, whose frames are copied in the step's
own stream: device memory, pinned host memory, one of each, one output only, a
sink off the 16-byte boundary (the copy engine), with a ring of host frames
shorter than the run.  Every frame is a deterministic function of the inputs, so
all agree with the pageable host sink bit for bit."""
import numpy as np
import pytest

from series_case import Case, instances, make_screens

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

CASE = Case(alt=[0.0, 1000.0, 5000.0], cn2=[0.6, 0.3, 0.1], speed=[8.0, 12.0, 20.0], direction=[0.0, 1.0, 2.5],
            sci=[(1.6e-6, 0.0, 0.0), (2.2e-6, 1e-5, 0.0)])
STEPS, SLOTS = 5, 3


def series(screens, amplitude, monkeypatch):
    from atmosphericturbulencesimul_gb300 import Series
    monkeypatch.setenv("ATMWFS_TILE_CFG", "2")  # one configuration: the autotuner could pick another per series
    c = Case(**{**CASE.__dict__, "amplitude": amplitude})
    s = Series(c.alt, c.cn2, c.speed, c.direction, master_size=c.M, instances=instances(c), pupil_scale=c.pupil,
               time_step=c.dt, fresnel_bin=c.fresnel_bin, zangle=c.zangle, amplitude=amplitude, fresnel=c.fresnel, ring=1)
    for l, sc in enumerate(screens):
        s.load_screen(l, sc)
    return s


@pytest.mark.parametrize("amplitude", [1, 0])
@pytest.mark.parametrize("pha_on,amp_on,off", [("cuda", "cuda", 0), ("pin", "pin", 0), ("cuda", "pin", 0), ("pin", "cuda", 0),
                                               ("cuda", None, 0), (None, "pin", 0), ("cuda", "cuda", 1)])
def test_in_stream_copies(lib, oracle64, monkeypatch, amplitude, pha_on, amp_on, off):
    screens = make_screens(CASE, oracle64)
    s = series(screens, amplitude, monkeypatch)
    n = SLOTS * s.frame_floats
    pha, amp = np.zeros(n, np.float32), np.zeros(n, np.float32)
    s.run(STEPS, pha=pha, amp=amp, nslots=SLOTS)
    s.close()
    assert np.isfinite(pha).all() and np.ptp(pha) > 0

    def sink(where):
        if where is None:
            return None
        return torch.zeros(n + 4, device="cuda") if where == "cuda" else torch.zeros(n + 4, pin_memory=True)

    s = series(screens, amplitude, monkeypatch)
    sp, sa = sink(pha_on), sink(amp_on)
    s.run(STEPS, pha_ptr=sp.data_ptr() + 4 * off if sp is not None else 0,
          amp_ptr=sa.data_ptr() + 4 * off if sa is not None else 0, nslots=SLOTS)
    s.close()
    for got, want in ((sp, pha), (sa, amp)):
        if got is not None:
            assert np.array_equal(got.cpu().numpy()[off:off + n], want)
