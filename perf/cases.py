"""The work whose speed counts, through the public entry points.

The paths, each over the range of sizes that this repository's benchmark,
tests and configurations use:

- "loop":   one or more RK2 steps of the Orszag-Tang vortex driven operator
            by operator, as a host time loop that calls the library in place
            of its own operators does;
- "vortex": the same vortex as fused RK2 steps (one CUDA graph per step);
- "torus":  the magnetised Kerr torus as fused RK2 steps, on grids from the
            parity tests' 24x16x8 to the benchmark's 192x96x64, with the time
            averages or the polar-axis correction in some;
- "radtorus": the radiative torus as RK2IMEX steps (two implicit and two
            explicit stages), with or without the warm-start network;
- "solve":  the batched implicit gas-radiation source solve on device cells,
            from the cell's own state or from the network's prediction;
- "u2p":    the MHD inversion of device cells;
- "forward", "train": inference and one epoch of training of the network.

A grid pass uploads the state from pinned host memory, runs its steps and
downloads the state, as a program that keeps its state on the host between
outputs does; so a pass always starts from the same state.
"""
import ctypes
import math

import numpy as np
import torch

import koral_b200 as k
from koral_b200 import train_warmstart as tw

SIGMA = (1e-3, 1e3)       # B^2/rho of magnetised cells, as the networks are trained on


def listed():
    return [
        # the smallest grid of the tests, one operator call after another:
        # launches and latency only
        dict(name="loop 16x16", path="loop", n=16, steps=4),
        # the small two-dimensional vortex between outputs: latency bound,
        # 16384 cells a kernel
        dict(name="vortex 128x128", path="vortex", n=128, steps=40),
        # a ragged small torus with the running time averages
        dict(name="torus 47x30x18 averages", path="torus", nx=47, ny=30, nz=18, steps=30, avg=True, polar=0),
        # the magnetised torus of the benchmark
        dict(name="torus 192x96x64", path="torus", nx=192, ny=96, nz=64, steps=10, avg=False, polar=0),
        # the parity tests' radiative torus, solver from the cell's own state
        dict(name="radtorus 24x16x8", path="radtorus", nx=24, ny=16, nz=8, steps=2, network=False),
        # the benchmark's default workload at half its resolution: radiative
        # torus with the learned warm start, past the worst of its transient
        dict(name="radtorus 128x64x32 network", path="radtorus", nx=128, ny=64, nz=32, steps=4, network=True),
        # a caller with few cells: latency of the longest cascade
        dict(name="solve 1537", path="solve", n=1537, sigma=False, network=False),
        # the batched solve of the benchmark, a sixteenth of its cells
        dict(name="solve 262144", path="solve", n=262144, sigma=False, network=False),
        # and from the network's prediction (features, network, solve)
        dict(name="solve 262144 network", path="solve", n=262144, sigma=True, network=True),
        # the MHD inversion of magnetised cells after a step has moved them
        dict(name="u2p 1048576", path="u2p", n=1048576, sigma=True),
        # the network on half the benchmark torus's cells
        dict(name="forward 1048576", path="forward", n=1048576),
        # an epoch of its training at the trainer's batch
        dict(name="train 262144", path="train", n=262144, batch=8192),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    path = rng.choice(["loop", "vortex", "torus", "torus", "radtorus", "solve", "solve", "u2p", "forward", "train"])
    if path == "loop":
        return dict(path=path, n=_log(rng, 16, 256), steps=rng.randint(1, 8))
    if path == "vortex":
        return dict(path=path, n=_log(rng, 16, 512), steps=rng.randint(4, 24))
    if path == "torus":
        nx, ny, nz = _log(rng, 24, 192), _log(rng, 16, 96), _log(rng, 8, 64)
        return dict(path=path, nx=nx, ny=ny, nz=nz, steps=rng.randint(2, 10), avg=rng.random() < .3 and nx * ny * nz < 60000,
                    polar=rng.choice([0, 0, k.POLAR_CORRECT]))
    if path == "radtorus":
        return dict(path=path, nx=_log(rng, 24, 112), ny=_log(rng, 16, 56), nz=_log(rng, 8, 28), steps=rng.randint(1, 4),
                    network=rng.random() < .5)
    if path == "solve":
        net = rng.random() < .5
        return dict(path=path, n=_log(rng, 100, 262144), sigma=net, network=net)
    if path == "u2p":
        return dict(path=path, n=_log(rng, 100, 1048576), sigma=rng.random() < .7)
    if path == "forward":
        return dict(path=path, n=_log(rng, 100, 1048576))
    return dict(path=path, n=_log(rng, 20000, 262144), batch=rng.choice([2048, 4096, 8192]))


# ---------------------------------------------------------------------------
# states
# ---------------------------------------------------------------------------
def _pinned(shape):
    return torch.empty(shape, dtype=torch.float64, pin_memory=True)


def _dp(t):
    return ctypes.cast(t.data_ptr(), ctypes.POINTER(ctypes.c_double))


def _grid_state(s, case):
    """The context, its state in pinned memory to start from, and room for
    what comes back."""
    u, p = s.download_state()
    st = dict(path=case["path"], s=s, steps=case["steps"], den=s.tstepdenmax,
              u0=torch.from_numpy(u).pin_memory(), p0=torch.from_numpy(p).pin_memory(), u=_pinned(s.shape),
              p=_pinned(s.shape), avg=bool(case.get("avg")))
    return st


def _vortex(case, seed):
    """The vortex with 1% noise on the gas energy, conserved state to match."""
    s = k.orszag_tang(case["n"])
    u, p = s.download_state()
    rng = np.random.default_rng(seed)
    p[..., 1] *= 1. + 0.01 * (rng.random(p.shape[:3]) - .5)
    g20, G20 = np.zeros((p[..., 0].size, 20)), np.zeros((p[..., 0].size, 20))
    for i, v in ((0, -1.), (6, 1.), (12, 1.), (18, 1.)):
        g20[:, i] = G20[:, i] = v
    g20[:, 19] = 1.
    u = k.p2u_cells(s.cfg, p.reshape(-1, s.nv), g20, G20).reshape(p.shape)
    s.upload_state(u, p)
    s.set_bc()
    s.begin_run()
    s.rk2_steps(2)      # past the first step, whose time step is the start-up one
    return s


def _rad_params():
    return k.rad_params()


def _to(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def prepare(case, seed):
    path = case["path"]
    if path in ("loop", "vortex"):
        return _grid_state(_vortex(case, seed), case)
    if path == "torus":
        s = k.fm_torus(case["nx"], case["ny"], case["nz"], k.torus_params(seed=seed))
        if case["polar"]:
            s.set_polar_correction(case["polar"])
        s.rk2_steps(4, graph=True)
        if case["avg"]:
            s.set_avg(True)
        return _grid_state(s, case)
    if path == "radtorus":
        s = k.radtorus(case["nx"], case["ny"], case["nz"], k.torus_params(seed=seed))
        mlp = tw.load(k, tw.DEFAULT_OUT_RADTORUS) if case["network"] else None
        s.set_implicit_solver(k.RAD_BATCHED, mlp)
        s.rk2imex_steps(12, graph=True)
        return _grid_state(s, case)
    if path == "solve":
        rp = _rad_params()
        uu, pp, g, G, dt = k.rad_cells(case["n"], seed, rp, sigma=SIGMA if case["sigma"] else None)
        opts = k.solver_opts()
        return dict(path=path, rp=rp, cells=[_to(a) for a in (uu, pp, g, G, dt)], opts=opts,
                    work=torch.empty(int(k.lib().kgpu_rad_work_bytes(case["n"])), dtype=torch.uint8, device="cuda"),
                    mlp=tw.load(k) if case["network"] else None)
    if path == "u2p":
        cells, _ = _u2p_cells(case, seed)
        return dict(path=path, cfg=k.u2p_config(_rad_params().gamma), cells=[_to(a) for a in cells])
    mlp = tw.load(k)
    X = _features(case["n"], seed)
    if path == "forward":
        return dict(path=path, mlp=mlp, X=X)
    # training goes on from the committed weights, on targets with noise
    gen = torch.Generator(device="cuda").manual_seed(seed)
    Y = mlp.forward(X)[:, :k.MLP_OUT]
    T = (Y + 0.1 * Y.std(0) * torch.randn(Y.shape, device="cuda", generator=gen)).contiguous()
    return dict(path=path, mlp=mlp, X=X, T=T, batch=case["batch"], epoch=0)


def _features(n, seed):
    """Network inputs: order one, as mlp_features scales them."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    return 1.5 * torch.randn((n, 16), device="cuda", generator=gen)


def _u2p_cells(case, seed):
    """Cells of the batched-solve distribution whose primitives a step has
    moved: the inversion starts from the primitives before it.  Gas Lorentz
    factors up to 20.  Returns ((uu, guess, g, G), the primitives)."""
    rp = _rad_params()
    uu, pp, g, G, _ = k.rad_cells(case["n"], seed, rp, sigma=SIGMA if case["sigma"] else None)
    rng = np.random.default_rng(seed + 1)
    guess = pp.copy()
    guess[:, 0] *= 1. + 0.02 * (rng.random(case["n"]) - .5)
    guess[:, 1] *= 10. ** rng.uniform(-.2, .2, case["n"])
    guess[:, 2:5] *= 1. + 0.02 * (rng.random((case["n"], 3)) - .5)
    return (uu, guess, g, G), pp


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def _rk2_loop(s):
    """One RK2 step operator by operator (the loop of ko.c:571-626)."""
    U, UT0, UT1, UT2 = k.ARR_U, k.ARR_UT0, k.ARR_UT1, k.ARR_UT2
    dt = s.begin_step()
    s.save_timesteps()
    s.copyi_u(1., U, UT0)
    s.do_correct()
    s.op_explicit(0., .5 * dt)
    s.calc_u2p()
    s.op_implicit(0., .5 * dt)
    s.copyi_u(1., U, UT1)
    s.op_explicit(0., dt)
    s.calc_u2p()
    s.op_implicit(0., dt)
    s.addi_u(1., U, -1., UT1, UT2)
    s.addi_u(1., UT0, 1., UT2, U)


def run(st):
    path = st["path"]
    if path in ("loop", "vortex", "torus", "radtorus"):
        s, L = st["s"], k.lib()
        k._check(L.kgpu_upload_state(s.h, _dp(st["u0"]), _dp(st["p0"])), "kgpu_upload_state")
        s.tstepdenmax = st["den"]
        if st["avg"]:
            s.reset_avg()
        if path == "loop":
            for _ in range(st["steps"]):
                _rk2_loop(s)
        elif path == "radtorus":
            s.rk2imex_steps(st["steps"], graph=True)
        else:
            s.rk2_steps(st["steps"], graph=True)
        k._check(L.kgpu_download_state(s.h, _dp(st["u"]), _dp(st["p"])), "kgpu_download_state")
        out = dict(u=st["u"], p=st["p"], den=s.tstepdenmax)
        if st["avg"]:
            out["avg"] = s.download_avg()[0]
        return out
    if path == "solve":
        uu, pp, g, G, dt = st["cells"]
        y = st["mlp"].forward(k.rad_features_device(st["rp"], pp, g, G, dt)) if st["mlp"] else None
        po, uo, status, attempt, iters, _ = k.rad_solve_device(st["rp"], uu, pp, g, G, dt, ypred=y, work=st["work"],
                                                               opts=st["opts"])
        return dict(pp=po, uu=uo, status=status, attempt=attempt, iters=iters)
    if path == "u2p":
        po, status, fixup, iters, _ = k.u2p_cells_device(st["cfg"], *st["cells"])
        return dict(pp=po, status=status, fixup=fixup, iters=iters)
    if path == "forward":
        return st["mlp"].forward(st["X"])
    st["epoch"] += 1
    loss = st["mlp"].train_epoch(st["X"], st["T"], batch=st["batch"], lr=1e-4, seed=st["epoch"])
    return dict(loss=loss, weights=st["mlp"].get())


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
# FP64 operations of the arithmetic itself, per cell: an MHD stage (three
# faces of 1.9 kFLOP, speeds, source, inversion, floors), a radiation stage's
# explicit part, one evaluation of the implicit residual
STAGE, STAGE_RAD, EVAL = 8000, 2500, 1500


def work(case):
    path = case["path"]
    if path in ("loop", "vortex", "torus", "radtorus"):
        nv = 13 if path == "radtorus" else 9
        n = case["n"] ** 2 if "n" in case else case["nx"] * case["ny"] * case["nz"]
        by = 4 * nv * 8 * n * (case["steps"] + 1)
        if path == "radtorus":     # four evaluations an iteration and a few iterations a solve, at the least
            return dict(bytes=by, flops=n * case["steps"] * 2 * (STAGE + STAGE_RAD + 12 * EVAL))
        return dict(bytes=by + (2 * 148 * 8 * n * case["steps"] if case.get("avg") else 0),
                    flops=n * case["steps"] * 2 * STAGE)
    n = case["n"]
    if path == "solve":
        return dict(bytes=n * (8 * (4 * 13 + 40 + 1) + 12), flops=n * 60 * EVAL)
    if path == "u2p":
        return dict(bytes=n * (8 * (3 * 9 + 40) + 12), flops=n * 800)
    layers = 2 * (16 * 128 + 128 * 128 + 128 * 8)
    if path == "forward":
        return dict(bytes=n * 4 * 24, flops=n * layers)
    return dict(bytes=n * 4 * (16 + 7) + 4 * 20000, flops=n * 3 * layers)


def tolerance(case):
    """About four times what one unit in the last place of the inputs makes
    of the outputs.  The flow has branches (floors, fixups, failed
    inversions) that amplify it: little on the vortex, much in the tori's
    atmosphere, and the implicit solve is ill-conditioned over part of its
    range.  The network is BF16."""
    return {
        "loop": dict(rel=1e-13, max=1e-12),
        "vortex": dict(rel=1e-13, max=1e-12),
        "torus": dict(rel=1e-4, max=2e-2),
        "radtorus": dict(rel=.03, max=.99),
        "solve": dict(rel=.03, max=.99, differ=.01),
        "u2p": dict(rel=3e-5, max=8e-3, differ=1e-5),
        "forward": dict(rel=1e-3, max=.3),
        "train": dict(rel=1e-3, max=3e-3),
    }[case["path"]]


# ---------------------------------------------------------------------------
# the outputs in 64 bits, without this repository's code
# ---------------------------------------------------------------------------
def exact(case, seed):
    path = case["path"]
    if path == "u2p":
        # the primitives that the conserved state was made from (nine MHD
        # variables; the others pass through)
        _, pp = _u2p_cells(case, seed)
        return dict(pp=pp, status=None, fixup=None, iters=None)
    if path == "forward":
        w = torch.from_numpy(np.load(tw.DEFAULT_OUT)["blob"].astype(np.float64)).cuda()
        at = np.cumsum([0, 16 * 128, 128, 128 * 128, 128, 128 * 8, 8, 8, 8])
        W1, b1, W2, b2, W3, b3, mean, scale = (w[at[i]:at[i + 1]] for i in range(8))
        a = _features(case["n"], seed).double()
        for W, c in ((W1, b1), (W2, b2)):
            z = a @ W.reshape(-1, 128) + c
            a = z * torch.sigmoid(z)
        return (a @ W3.reshape(128, 8) + b3) * scale + mean
    # the grid steps would need a second general-relativistic MHD code; the
    # implicit solve stops on a residual test, and over part of its range one
    # unit in the last place of the input moves the result by order one; an
    # epoch of training depends on its shuffling
    return None
