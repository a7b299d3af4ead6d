"""The MHD inversion of device cells (k_u2p_first, k_u2p_rest) against the
one-thread-per-cell inversion of kgpu_u2p_cells, bit for bit, at the sizes
where its ranges and lists can go wrong (one cell, a part-filled warp, one
more than a block, one more than a range of the second launch) and from
guesses near and far: the far ones send a large share of the cells to the
second launch, to both equations and to failure."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# 310001: ranges of the largest size, 1024 cells, and a last one that is not full
@pytest.mark.parametrize("n, far", [(n, far) for n in (1, 31, 129, 4097, 40001) for far in (0.02, 1.0, 6.0)] +
                         [(310001, 1.0)])
def test_device_cells_equal_one_thread_per_cell(kgpu, n, far):
    import torch
    rp = kgpu.rad_params()
    cfg = kgpu.u2p_config(rp.gamma)
    uu, pp, g, G, _ = kgpu.rad_cells(n, n, rp, sigma=(1e-3, 1e3))
    rng = np.random.default_rng(n)
    pp[:, 1] *= 10. ** rng.uniform(-far, far, n)
    pp[:, 2:5] *= 1. + far * (rng.random((n, 3)) - .5)
    uu[:, 1] *= 1. + .1 * far * rng.uniform(-1, 1, n)
    uu[rng.random(n) < .01, 0] *= -1.
    a = [np.ascontiguousarray(x) for x in (uu[:, :9], pp[:, :9], g, G)]
    ph, sh, fh = kgpu.u2p_cells(cfg, *a)
    pd, sd, fd, it, stats = kgpu.u2p_cells_device(cfg, *[torch.from_numpy(x).cuda() for x in a])
    assert np.array_equal(sd.cpu().numpy(), sh) and np.array_equal(fd.cpu().numpy(), fh)
    assert np.array_equal(pd.cpu().numpy().view(np.int64), ph.view(np.int64))
    assert stats[0] == int(it.sum())
