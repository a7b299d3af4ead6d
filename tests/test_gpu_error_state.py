"""A call that fails on the host leaves nothing behind: after a context that
does not fit the device's memory, an inversion stage of another context runs
to its end (all its launches, its work queues emptied) and gives the bits of a
context that saw no failure."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_failed_allocation_leaves_later_calls_alone(kgpu):
    out = []
    for fail in (False, True):
        s = kgpu.fm_torus(24, 16, 8)
        u, p = s.download_state()
        rng = np.random.default_rng(0)
        u[rng.random(u.shape[:3]) < .02, 0] *= -1.     # cells that ask for the neighbour fixup
        s.upload_state(u, p)
        if fail:
            with pytest.raises(kgpu.KgpuError):
                kgpu.Subdomain(kgpu.default_config(200000, 20000, 100))   # 29 TB an array
        for _ in range(2):
            s.calc_u2p()
        out.append(s.download_state())
        assert s.counters()["fixups"] > 0
    for a, b in zip(*out):
        assert np.array_equal(a.view(np.int64), b.view(np.int64))
