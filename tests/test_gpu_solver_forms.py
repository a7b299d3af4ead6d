"""The implicit solver's forms and options inside the step of the radiative
torus (24x16x8, built by the library itself): every form and option gives the
same bits, from the stream and from a CUDA graph, and options belong to the
context they are set on."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def start(kgpu, mode, warm=None, **opts):
    s = kgpu.radtorus(24, 16, 8)
    s.set_implicit_solver(mode, warm)
    if opts:
        s.set_implicit_options(**opts)
    return s


def same(a, b):
    return all(np.array_equal(x.view(np.int64), y.view(np.int64)) for x, y in zip(a, b))


def test_solver_forms_and_graph_identical(kgpu):
    """inner_cap: the evaluations of a nested inversion in one lane before a
    whole warp takes it (0: never); thin: the persistent form's hand-over."""
    ref = None
    for mode, graph, opts in ((kgpu.RAD_PLAIN, False, {}), (kgpu.RAD_PLAIN, True, {}), (kgpu.RAD_BATCHED, False, {}),
                              (kgpu.RAD_BATCHED, True, {}), (kgpu.RAD_BATCHED, True, dict(inner_cap=4)),
                              (kgpu.RAD_BATCHED, False, dict(inner_cap=0)), (kgpu.RAD_PERSISTENT, False, {}),
                              (kgpu.RAD_PERSISTENT, True, dict(thin=0)),
                              (kgpu.RAD_PERSISTENT, True, dict(thin=32, inner_cap=4))):
        s = start(kgpu, mode, **opts)
        s.rk2imex_steps(3, graph=graph)
        out = s.download_state()
        c = s.counters()
        got = (c["imp_iters"], c["imp_evals"], c["imp_solves"], c["radimp_failed"])
        if ref is None:
            ref = out, got
        assert same(ref[0], out) and ref[1] == got, (mode, graph, opts)
        # the option reaches the solver: only a cap hands evaluations to a warp
        if mode == kgpu.RAD_BATCHED:
            assert (c["imp_cooperative"] == 0) == (opts.get("inner_cap") == 0)
        s.close()


def test_solver_options_per_context(kgpu):
    """Two contexts in one process hold their own solver: setting one leaves
    the other alone, a captured step graph is captured anew when its context's
    options change (its launches and counters follow them), and the results
    stay the same bits."""
    a, b = (start(kgpu, kgpu.RAD_BATCHED) for _ in range(2))
    a.set_implicit_solver(kgpu.RAD_PERSISTENT, None)
    assert (a.tuning().implicit_mode, b.tuning().implicit_mode) == (kgpu.RAD_PERSISTENT, kgpu.RAD_BATCHED)
    b.set_implicit_options(inner_cap=8)
    assert (a.implicit_options().inner_cap, b.implicit_options().inner_cap) == (kgpu.solver_opts().inner_cap, 8)

    def step(s):
        n = s.launches
        s.reset_counters()
        s.rk2imex_steps(1, graph=True)
        return s.launches - n, s.counters()["imp_cooperative"]

    la, _ = step(a)
    lb, handed = step(b)
    # one launch fewer in each of the two solves
    assert lb - la == 2 and handed > 0
    a.set_implicit_solver(kgpu.RAD_BATCHED, None)   # between two graph steps
    b.set_implicit_options(inner_cap=0)
    la, handed_a = step(a)
    assert step(b) == (la, 0) and la == lb and handed_a > 0
    assert same(a.download_state(), b.download_state())
    with pytest.raises(kgpu.KgpuError):
        a.set_implicit_options(thin=33)


def test_warm_attempts_reach_a_captured_step(kgpu):
    """With a network: how many attempts a cell may run from its prediction is
    read by the step captured after it was set."""
    from koral_b200 import train_warmstart as tw
    mlp = tw.load(kgpu, tw.DEFAULT_OUT_RADTORUS)
    s = start(kgpu, kgpu.RAD_BATCHED, mlp)
    u, p = s.download_state()
    den = s.tstepdenmax
    seen = []
    for attempts in (6, 1, 6):
        s.set_implicit_options(warm_attempts=attempts)
        s.upload_state(u, p)
        s.tstepdenmax = den
        s.reset_counters()
        s.rk2imex_steps(1, graph=True)
        seen.append(s.counters()["imp_fallbacks"])
    assert seen[0] == seen[2] < seen[1]
