"""MP5's limiters by sign tests (kgpu_physics.cuh) against the reference's
products of signs (finite.c:226-286) restated in numpy, bit for bit, on the
CPU: stencils of either slope, with equal values and zeros of both signs, near
the ends of the range (where the products are kept), with infinities and NaN."""
import ctypes

import numpy as np
import pytest

from test_host_physics import P, host, pytestmark  # noqa: F401  (the harness and its skip)


def sign(x):
    return np.where(x > 0., 1., np.where(x < 0., -1., np.where(x == 0., 1., 0.)))


def dmin(a, b):
    return np.where(a < b, a, b)


def dmax(a, b):
    return np.where(a > b, a, b)


def dmm(x, y):
    return .5 * (sign(x) + sign(y)) * dmin(abs(x), abs(y))


def dm4(w, x, y, z):
    return (0.125 * (sign(w) + sign(x)) * abs((sign(w) + sign(y)) * (sign(w) + sign(z))) *
            dmin(dmin(abs(w), abs(x)), dmin(abs(y), abs(z))))


def mp5(um2, um1, u0, up1, up2):
    vor = (3. * um2 - 20. * um1 + 90. * u0 + 60. * up1 - 5. * up2) / 128.
    vmp = u0 + dmm(up1 - u0, 4. * (u0 - um1))
    djm1, dj, djp1 = um2 - 2. * um1 + u0, um1 - 2. * u0 + up1, u0 - 2. * up1 + up2
    ph = dm4(4. * dj - djp1, 4. * djp1 - dj, dj, djp1)
    mh = dm4(4. * dj - djm1, 4. * djm1 - dj, dj, djm1)
    vul, vav = u0 + 4. * (u0 - um1), 0.5 * (u0 + up1)
    vmd, vlc = vav - 0.5 * ph, u0 + 0.5 * (u0 - um1) + 1.3333333 * mh
    vmin = dmax(dmin(u0, dmin(up1, vmd)), dmin(u0, dmin(vul, vlc)))
    vmax = dmin(dmax(u0, dmax(up1, vmd)), dmax(u0, dmax(vul, vlc)))
    return np.where((vor - u0) * (vor - vmp) < 1.e-10, vor, vor + dmm(vmin - vor, vmax - vor))


def stencils(kind, n=100000):
    rng = np.random.default_rng(5)
    u = rng.normal(size=(n, 5))
    if kind == "sorted":
        u = np.sort(u, axis=1) * rng.choice([-1., 1.], (n, 1))
    elif kind == "steep":
        u = np.exp(8. * u)
    elif kind == "equal":
        u = np.round(u)
        z = u == 0.
        u[z] = rng.choice([0., -0.], z.sum())
    elif kind == "huge":
        u = u * 10. ** rng.uniform(295, 308, (n, 1))
    elif kind == "special":
        m = rng.random(u.shape)
        u[m < .05], u[(m > .05) & (m < .1)], u[(m > .1) & (m < .15)] = np.nan, np.inf, -np.inf
    return np.ascontiguousarray(u)


@pytest.mark.parametrize("kind", ["normal", "sorted", "steep", "equal", "huge", "special"])
def test_mp5_sign_tests(host, kind):  # noqa: F811
    u = stencils(kind)
    left, right = np.zeros(len(u)), np.zeros(len(u))
    host.hp_recon(ctypes.c_long(len(u)), 4, P(u), P(np.ones_like(u)), P(left), P(right))
    with np.errstate(all="ignore"):
        for got, want in ((right, mp5(*u.T)), (left, mp5(*u.T[::-1]))):
            nan = np.isnan(want)
            assert np.array_equal(np.isnan(got), nan)
            assert np.array_equal(got[~nan].view(np.int64), want[~nan].view(np.int64))
