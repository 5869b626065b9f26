"""Phase-only frames in both launch shapes: an instance's frames do not depend
on which other instances the context holds.  Alone (two rows per CTA, one job),
as one of more wavelengths of its direction than fit in shared memory at a time
(the group dealt to several jobs), and as one of a fan of directions large
enough for eight rows per CTA; one layer and several; Scoeff equal on all
layers and not; a crop off the row tiles.

The same samples and sums in the same order: bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def frames(lib, inst, L, screens, nsteps=2):
    from atmosphericturbulencesimul_gb300 import Series
    s = Series([1000.0 * (k + 1) for k in range(L)], [1.0] * L, [5.0 + 3 * k for k in range(L)],
               [0.7 * k for k in range(L)], master_size=screens[0].shape[0], instances=inst, pupil_scale=0.02,
               time_step=1e-3, amplitude=0)
    for l in range(L):
        s.load_screen(l, screens[l])
    out = s.run_frames(nsteps)
    s.close()
    return out


@pytest.mark.parametrize("W,crop,L,fan,even", [
    (64, 64, 1, 40, True), (64, 61, 7, 40, False), (128, 100, 3, 24, True), (256, 255, 7, 8, True),
    (256, 256, 16, 8, False), (512, 509, 2, 3, True),
])
def test_frames_do_not_depend_on_the_launch_shape(lib, W, crop, L, fan, even):
    from atmosphericturbulencesimul_gb300 import InstanceSpec
    rng = np.random.default_rng(W + L)
    screens = [np.cumsum(rng.standard_normal((512, 512)), 0).astype(np.float32) * 1e-8 for _ in range(L)]

    def inst(q, d):
        sc = np.full(L, 1.0 + 0.01 * q, np.float32)
        if not even:
            sc += np.linspace(0, 0.1, L).astype(np.float32)
        return InstanceSpec(lam=1e-6 + 1e-8 * q, wf_raw_size=W, wf_size=crop, src_x=2e-5 * d, src_y=-1e-5 * d, scoeff=sc)

    colours = frames(lib, [inst(q, 1) for q in range(40)], L, screens)
    fans = frames(lib, [inst(3, d) for d in range(fan)], L, screens)
    for q, d, got in ((0, 1, colours[0]), (33, 1, colours[33]), (39, 1, colours[39]), (3, 1, colours[3]), (3, 1, fans[1]),
                      (3, fan - 1, fans[fan - 1])):
        alone = frames(lib, [inst(q, d)], L, screens)[0]
        assert np.isfinite(got[0]).all() and np.ptp(got[0]) > 0
        assert np.array_equal(got[0], alone[0]) and np.array_equal(got[1], alone[1]), (q, d)
