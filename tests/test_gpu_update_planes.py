"""The update step with the Christoffel rows of an axisymmetric metric shared
between the four planes of a block, against the same grid with the metric
stored for every plane (each cell loads its own rows), bit for bit: planes that
fill the last block and planes that do not, a plane that ends inside a warp, the
launch bounds that the tuning offers, and the grids that keep their own rows
(fewer than four planes, few blocks)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(21, 11, 5), (192, 96, 3), (160, 72, 4), (131, 61, 9), (190, 95, 10)])
def test_shared_rows_equal_own_rows(kgpu, shape):
    out = []
    for axisym in (1, 0):
        cfg = kgpu.torus_config(*shape)
        cfg.axisym_metric = axisym
        s = kgpu.Subdomain(cfg)
        s.init_fm_torus(None, on_host=True)
        for blocks in (3, 4, 5):
            t = s.tuning()
            t.update_blocks = blocks
            s.set_tuning(t)
            s.rk2_steps(2)
        out.append(s.download_state())
    for a, b in zip(*out):
        assert np.array_equal(np.asarray(a).view(np.int64), np.asarray(b).view(np.int64))
