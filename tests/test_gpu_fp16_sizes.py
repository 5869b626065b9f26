"""FP16 transforms at every grid size (their passes take tile configuration 2 of
the size, and at 2048 the three-stage plan) against the FP64 oracle: λref and a
science instance, two hops, a crop off the row tiles.

Bars: those of the precision study (test_gpu_precision.py), every frame within
3 nm rms wrapped OPD error and 1e-2 relative amplitude variance."""
import numpy as np
import pytest

from series_case import Case, instances, make_screens, metrics, run_oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W,Wout", [(64, 64), (128, 101), (256, 255), (1024, 1000), (2048, 2001)])
def test_fp16_transforms(lib, oracle64, W, Wout):
    from atmosphericturbulencesimul_gb300 import Series
    case = Case(alt=[0.0, 2000.0, 9000.0], cn2=[0.6, 0.25, 0.15], speed=[8.0, 12.0, 20.0], direction=[0.0, 1.0, 2.5],
                M=max(256, W), W=W, Wout=Wout, sci=[(1.25e-6, 0.0, 0.0)])
    screens = make_screens(case, oracle64)
    inst = instances(case)
    s = Series(case.alt, case.cn2, case.speed, case.direction, master_size=case.M, instances=inst, pupil_scale=case.pupil,
               time_step=case.dt, fresnel_bin=case.fresnel_bin, fft_fp16=1)
    for l, sc in enumerate(screens):
        s.load_screen(l, sc)
    frames = s.run_frames(1)
    s.close()
    _, res, _, _ = run_oracle(case, oracle64, screens, 1)
    for i, I in enumerate(inst):
        pha_o, amp_o = res[0][i]
        m = metrics(frames[i][0][0], frames[i][1][0], pha_o, amp_o, I.lam)
        assert m["wrapped_rms_nm"] < 3.0, m
        assert amp_o.var() < 1e-6 or m["amp_var_rel"] < 1e-2, m
