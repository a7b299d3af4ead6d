"""The face fluxes of all directions in one launch (small grids), against the
launches by direction, which the split form takes at every size, bit for bit:
fluxes, EMFs and the updated state, with and without faces that need the
magnetic floor, with radiation, and on grids of few planes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def run(kgpu, make, split):
    s = make()
    t = s.tuning()
    t.flux_split = split
    s.set_tuning(t)
    s.profile(True)
    s.profile_reset()
    s.op_explicit(0., 1e-3)
    s.profile(False)
    prof = s.profile_read()
    assert prof["k_flux_all"][1] == (0 if split else 1)
    if s.cfg.nv == 13:
        assert prof["k_flux_rad_all"][1] == (0 if split else 1)
    out = [*s.download_state(), *[s.download_flux(d) for d in range(3)], s.download_emf()]
    return out, s.counters()["face_floors"]


@pytest.mark.parametrize("shape", [(24, 16, 8), (37, 11, 5), (30, 9, 4), (20, 9, 3), (21, 13, 2)])
@pytest.mark.parametrize("kind", ["torus", "floor", "rad"])
def test_one_launch_equals_launches_by_direction(kgpu, kind, shape):
    def make():
        if kind == "rad":
            s = kgpu.radtorus(*shape)
        else:
            cfg = kgpu.torus_config(*shape)
            if kind == "floor":
                cfg.b2rhoratiomax = 1e-5
            s = kgpu.Subdomain(cfg)
            s.init_fm_torus(None)
        u, p = s.download_state()
        p[..., 1] *= 1. + .2 * (np.random.default_rng(1).random(p.shape[:3]) - .5)   # no two neighbours alike
        s.upload_state(u, p)
        return s

    (a, fa), (b, fb) = run(kgpu, make, 0), run(kgpu, make, 1)
    assert fa == fb and (fa > 0) == (kind == "floor")
    for x, y in zip(a, b):
        x, y = np.ascontiguousarray(x), np.ascontiguousarray(y)
        assert np.array_equal(x.view(np.int64), y.view(np.int64))
