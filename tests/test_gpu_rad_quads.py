"""The batched implicit solve (four lanes a cell, work lists by kind of
attempt) against the other forms, bit for bit, at the sizes where its lists
and its lanes can go wrong: fewer cells than a warp takes, one cell a warp,
the last warp part-filled, as many cells as the chip holds warps and one more
(where the warps of a block begin to go in step), and enough cells that every
quad takes several.

* From the cells' own guess: the one-thread-per-cell form, results and the
  counters of Newton iterations and evaluations, whatever the cap on the
  evaluations of a nested inversion in one lane (each hands over to the whole
  warp at another point; 0: never).
* From the network's prediction: the persistent form, for every rule of where
  a warm-started cascade begins and after how many attempts it gives way to
  the reference's, which takes cells through every list in every order.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
SIGMA = (1e-3, 1e3)


def device_cells(kgpu, n, sigma):
    import torch
    rp = kgpu.rad_params()
    return rp, [torch.from_numpy(np.ascontiguousarray(a)).cuda()
                for a in kgpu.rad_cells(n, 100 + n, rp, sigma=sigma)]


def assert_same(a, b):
    import torch
    for x, y in zip(a[:5], b[:5]):
        if x.dtype == torch.float64:
            x, y = x.view(torch.int64), y.view(torch.int64)
        assert torch.equal(x, y)


@pytest.mark.parametrize("sigma", [None, SIGMA])
@pytest.mark.parametrize("n", [1, 3, 33, 1201, 2368, 2369, 21001])
def test_quads_equal_plain(kgpu, n, sigma):
    rp, d = device_cells(kgpu, n, sigma)
    a = kgpu.rad_solve_device(rp, *d, mode=kgpu.RAD_PLAIN, nstats=7)
    for cap in (64, 4, 0):
        b = kgpu.rad_solve_device(rp, *d, mode=kgpu.RAD_BATCHED, nstats=7, opts=kgpu.solver_opts(inner_cap=cap))
        assert_same(a, b)
        assert (a[5][0], a[5][3]) == (b[5][0], b[5][3])


@pytest.mark.parametrize("n", [33, 5003])
def test_warm_quads_equal_persistent(kgpu, n):
    from koral_b200 import train_warmstart as tw
    rp, d = device_cells(kgpu, n, SIGMA)
    y = tw.load(kgpu).forward(kgpu.rad_features_device(rp, *d[1:]))
    for skip in (0, 1, 2):
        for attempts in (6, 3, 2, 1):
            o = kgpu.solver_opts(skip=skip, warm_attempts=attempts)
            a = kgpu.rad_solve_device(rp, *d, mode=kgpu.RAD_PERSISTENT, ypred=y, nstats=7, opts=o)
            b = kgpu.rad_solve_device(rp, *d, mode=kgpu.RAD_BATCHED, ypred=y, nstats=7, opts=o)
            assert_same(a, b)
            assert (a[5][0], a[5][2], a[5][3]) == (b[5][0], b[5][2], b[5][3]), (skip, attempts)
