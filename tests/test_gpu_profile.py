"""A profiled step launches what a step without profiling does, and every
launch is in the profile: on a small grid (the three directions of the face
flux in one launch), on a larger one, with the face states reconstructed by a
kernel of their own, and with radiation."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("make, split", [
    (lambda k: k.orszag_tang(16), 0), (lambda k: k.fm_torus(24, 16, 8), 0), (lambda k: k.fm_torus(24, 16, 8), 1),
    (lambda k: k.fm_torus(120, 60, 20), 0), (lambda k: k.radtorus(24, 16, 8), 0)])
def test_profiled_step_is_the_step(kgpu, make, split):
    s = make(kgpu)
    t = s.tuning()
    t.flux_split = split
    s.set_tuning(t)
    step = s.rk2imex_steps if s.cfg.nv == 13 else s.rk2_steps
    step(1)
    n0 = s.launches
    step(1)
    n1 = s.launches
    s.profile(True)
    s.profile_reset()
    step(1)
    s.profile(False)
    assert s.launches - n1 == n1 - n0
    p = s.profile_read()
    dirs = 2 if s.cfg.nz == 1 else 3
    merged = not split and (s.cfg.nx < 100)
    assert p["k_flux_all"][1] == (2 if merged else 0)
    assert [p[f"k_flux_{a}"][1] for a in "xyz"[:dirs]] == [0 if merged else 2] * dirs
    assert p["k_flux_fix"][1] == (0 if split else 2)
    if s.cfg.nv == 13:
        assert p["k_flux_rad_all"][1] == 2 and p["k_flux_rad_x"][1] == 0
    else:
        # one record a launch; two launches share one with the split form's
        # floor pass
        assert sum(c for _, c in p.values()) + (2 * dirs if split else 0) == n1 - n0
