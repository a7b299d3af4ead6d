"""The rows of counters that calls of kgpu_u2p_cells_device hold while they
run: the bookkeeping on the CPU (no row in two hands, none lost, -1 when all
are held), and on the GPU calls of many threads, each on its own stream, which
must report the counters that they report one at a time."""
import ctypes
import os
import subprocess
import threading

import numpy as np
import pytest

from conftest import ROOT


@pytest.fixture(scope="module")
def host(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("slots") / "libslots.so")
    subprocess.check_call(["g++", "-O2", "-std=c++17", "-pthread", "-shared", "-fPIC", "-o", so,
                           os.path.join(ROOT, "tests", "slots", "slots_host.cc")])
    L = ctypes.CDLL(so)
    L.slots_collisions.restype = ctypes.c_long
    return L


def test_slots_one_holder(host):
    assert host.slots_all_distinct() == 1
    for threads in (2, 8, 96):
        assert host.slots_collisions(threads, 20000) == 0


@pytest.mark.gpu
@pytest.mark.parametrize("threads", [4, 80])
def test_counters_of_concurrent_calls(kgpu, threads):
    import torch
    rp = kgpu.rad_params()
    cfg = kgpu.u2p_config(rp.gamma)
    cells, alone = [], []
    for t in range(4):
        uu, pp, g, G, _ = kgpu.rad_cells(3000 + 700 * t, t, rp, sigma=(1e-3, 1e3))
        pp = pp.copy()
        pp[:, 1] *= 10. ** np.random.default_rng(t).uniform(-1, 1, len(pp))
        cells.append([torch.from_numpy(np.ascontiguousarray(x)).cuda() for x in (uu[:, :9], pp[:, :9], g, G)])
        alone.append(kgpu.u2p_cells_device(cfg, *cells[-1])[4])
    torch.cuda.synchronize()
    got = [[] for _ in range(threads)]

    def work(t):
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(5):
                got[t].append(kgpu.u2p_cells_device(cfg, *cells[t % 4])[4])

    ts = [threading.Thread(target=work, args=(t,)) for t in range(threads)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert all(got[t] == [alone[t % 4]] * 5 for t in range(threads))
