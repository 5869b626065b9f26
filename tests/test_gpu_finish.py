"""The step's last kernel in a context of one grid class (unwrap, apply and
step counter together) against the separate kernels that contexts of several
classes run: the same instances, alone and beside an instance of another grid,
give the same bits and the same relaxation counts, over steps with a window
advance between them.  Crops with no bin, one, and the most and one more than
the kernel takes; seeing that fires no vote, some, and up to the iteration
limit."""
import numpy as np
import pytest

from series_case import Case, make_screens, scoeff_for

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,Wout,seeing", [
    (64, 64, 0.7), (64, 19, 0.7), (64, 39, 3.0), (128, 100, 6.0), (256, 255, 3.0), (512, 512, 0.7), (512, 510, 4.0),
    (1024, 659, 2.0), (1024, 660, 0.7),
])
def test_finish_kernel_matches_separate_kernels(lib, oracle64, monkeypatch, W, Wout, seeing):
    from atmosphericturbulencesimul_gb300 import MODE_REF, MODE_SCI, InstanceSpec, Series
    monkeypatch.setenv("ATMWFS_TILE_CFG", "1")   # the same roundings in both contexts
    case = Case(alt=[0.0, 4000.0, 12000.0], cn2=[0.3, 0.3, 0.4], speed=[10.0, 20.0, 30.0], direction=[0.5, 2.0, 4.0],
                M=256, W=W, Wout=Wout, seeing=seeing)
    screens = make_screens(case, oracle64)
    spec = lambda lam, mode, w, wo: InstanceSpec(lam=lam, mode=mode, wf_raw_size=w, wf_size=wo, scoeff=scoeff_for(case, lam))
    own = [spec(0.5e-6, MODE_SCI, W, Wout), spec(0.5e-6, MODE_REF, W, Wout), spec(1.6e-6, MODE_SCI, W, Wout)]
    other = 64 if W != 64 else 128

    def frames(specs):
        s = Series(case.alt, case.cn2, case.speed, case.direction, master_size=case.M, instances=specs,
                   pupil_scale=case.pupil, time_step=case.dt, fresnel_bin=case.fresnel_bin)
        for l, scr in enumerate(screens):
            s.load_screen(l, scr)
        out, iters = [], []
        for _ in range(2):
            out.append([(p.copy(), a.copy()) for p, a in s.run_frames(2)[:3]])
            iters.append([s.last_iters(i) for i in (0, 2)])
            s.advance(1)
        assert s.steps_done == 6
        n = s.step_kernels()
        s.close()
        return out, iters, n

    a, ia, na = frames(own)
    b, ib, nb = frames(own + [spec(1.0e-6, MODE_SCI, other, other)])
    if Wout // 20 <= 32:
        assert na < nb - 7          # no unwrap, apply and counter of its own
    if Wout >= 20:
        assert ia == ib
    for fa, fb in zip(a, b):
        for (pa, aa), (pb, ab) in zip(fa, fb):
            assert np.array_equal(pa, pb) and np.array_equal(aa, ab)
