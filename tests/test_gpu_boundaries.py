"""The ghost cells, which one launch fills from domain cells alone, against
the rules of the reference written out in numpy pass by pass: the faces
(finite.c:2673-2748), then in 2D the periodic corners (3075-3328), in 3D the
edges along z, y and x and the corner blocks (3330-3705), each pass reading
what the ones before wrote.  Primitives bit for bit in the whole array (cells
that no rule fills keep their contents), conserved ones bit for bit against
p2u of those primitives, or the copy where the boundary copies them."""
import itertools

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def ghosts(kgpu, p, u, n, ng, bc):
    """The passes on arrays [z][y][x][variable]; returns which ghost cells
    were written with p2u and which with copies of u."""
    off = [ng if m > 1 else 0 for m in n]
    put = np.zeros(p.shape[:3], dtype=bool)
    idx = lambda c: (c[2] + off[2], c[1] + off[1], c[0] + off[0])

    def mean(t, a, b=None):
        p[idx(t)] = p[idx(a)] if b is None else .5 * (p[idx(a)] + p[idx(b)])
        put[idx(t)] = True

    for c in itertools.product(*[range(-o, m + o) for o, m in zip(off, n)]):
        out = [d for d in range(3) if not 0 <= c[d] < n[d]]
        if len(out) != 1:
            continue
        d, i, m = out[0], c[out[0]], n[out[0]]
        if bc[d] == kgpu.BC_OUTFLOW:
            src = 0 if i < 0 else m - 1
        elif bc[d] == kgpu.BC_REFLECT:
            src = -i - 1 if i < 0 else 2 * m - i - 1
        else:
            src = 0 if d > 0 and m < ng else i + m if i < 0 else i - m
        s = list(c)
        s[d] = src
        v = p[idx(s)].copy()
        if bc[d] == kgpu.BC_REFLECT:
            for q in (2, 6, 10)[:2 if v.size == 9 else 3]:
                v[q + d] = -v[q + d]
        p[idx(c)] = v
        put[idx(c)] = bc[d] != kgpu.BC_PERIODIC_COPY
        if bc[d] == kgpu.BC_PERIODIC_COPY:
            u[idx(c)] = u[idx(s)]
    edges = []
    if n[1] > 1:
        edges = [(2, 0, 1)] + ([(1, 0, 2), (0, 1, 2)] if n[2] > 1 else [])
    for c, a, b in edges:
        NA, NB = n[a], n[b]
        for t in range(-off[c], n[c] + off[c]):
            def at(va, vb):
                r = [0, 0, 0]
                r[a], r[b], r[c] = va, vb, t
                return r
            for hiA, hiB in itertools.product((0, 1), (0, 1)):
                gA, gB, iA, iB = NA if hiA else -1, NB if hiB else -1, NA - 1 if hiA else 0, NB - 1 if hiB else 0
                for i in range(ng - 1):
                    ta, tb = NA + i + 1 if hiA else -ng + i, NB + i + 1 if hiB else -ng + i
                    mean(at(ta, gB), at(ta, iB))
                    mean(at(gA, tb), at(iA, tb))
                sA, sB = 1 if hiA else -1, 1 if hiB else -1
                for j in range(2):
                    ta, tb = gA + j * sA, gB + j * sB
                    if n[2] == 1:
                        mean(at(ta, tb), at(j if hiA else NA - 1 - j, tb), at(j if hiA else NA - 1 - j, tb))
                    else:
                        mean(at(ta, tb), at(ta, tb - sB), at(ta - sA, tb))
    if n[1] > 1 and n[2] > 1:
        for hi in itertools.product((0, 1), repeat=3):
            for o in itertools.product(range(ng), repeat=3):
                mean([m + k if h else k - ng for h, k, m in zip(hi, o, n)], [m - 1 if h else 0 for h, m in zip(hi, n)])
    return put


def make(kgpu, n, bc, ng, nv):
    if n[1] > 1 and n[2] > 1:
        cfg = (kgpu.radtorus_config if nv == 13 else kgpu.torus_config)(*n)
        cfg.ng, cfg.axisym_metric = ng, 0
        for d in range(3):
            cfg.bc[d] = bc[d]
        s = kgpu.Subdomain(cfg)
        if nv == 13:
            import ctypes
            s._rp = kgpu.rad_params(mass=kgpu.RADTORUS_MASS, gamma=13. / 9.)
            kgpu._check(kgpu.lib().kgpu_init_fm_radtorus(s.h, ctypes.byref(kgpu.torus_params()), ctypes.byref(s._rp),
                                                         kgpu.RADTORUS_ERADATM, 0), "kgpu_init_fm_radtorus")
        else:
            s.init_fm_torus(None)
        return s
    s = kgpu.Subdomain(kgpu.default_config(*n, ng=ng, bc=bc))
    s.set_uniform_grid([0., 0., 0.], [1., 1., 1.])
    s.set_minkowski_metric()
    return s


def cases(kgpu_bc=(1, 2, 0, 3)):
    O, R, P, C = kgpu_bc
    for nv, ng in ((9, 4), (9, 5), (13, 4)):
        for bc in ((O, R, C), (R, R, R), (O, O, O), (P, P, P), (C, C, C), (R, O, P)):
            yield (9, 7, 6), bc, ng, nv
    for n in ((9, 7, 6), (5, 2, 3)):
        yield n, (O, P, P), 4, 9
        yield n, (R, O, O), 4, 9
    for n in ((7, 6, 1), (5, 3, 1), (3, 2, 1)):
        yield n, (P, P, P), 3, 9
    for bc in ((P, P, P), (O, R, R), (R, O, C), (C, P, O)):
        yield (8, 1, 1), bc, 3, 9
        yield (8, 1, 5), bc, 3, 9


@pytest.mark.parametrize("n, bc, ng, nv", list(cases()))
def test_ghost_cells(kgpu, n, bc, ng, nv):
    s = make(kgpu, n, bc, ng, nv)
    rng = np.random.default_rng(sum(n))
    p = np.empty(s.shape)
    p[..., 0] = rng.uniform(.1, 1., s.shape[:3])
    p[..., 1] = rng.uniform(.01, .1, s.shape[:3])
    p[..., 2:5] = .1 * rng.uniform(-1, 1, s.shape[:3] + (3,))
    p[..., 5:9] = .1 * rng.uniform(-1, 1, s.shape[:3] + (4,))
    if nv == 13:
        p[..., 9] = rng.uniform(.01, .1, s.shape[:3])
        p[..., 10:13] = .1 * rng.uniform(-1, 1, s.shape[:3] + (3,))
    u = rng.normal(size=s.shape)
    s.upload_state(u, p)
    s.set_bc()
    gu, gp = s.download_state()
    put = ghosts(kgpu, p, u, n, ng, bc)
    assert np.array_equal(gp.view(np.int64), p.view(np.int64))
    g, G = (np.ascontiguousarray(a.reshape(-1, 20)[put.ravel()]) for a in s.download_metric()[:2])
    q = np.ascontiguousarray(p[put])
    u[put] = kgpu.rad_p2u_cells(s._rp, q, g, G) if nv == 13 else kgpu.p2u_cells(s.cfg, q, g, G)
    assert np.array_equal(gu.view(np.int64), u.view(np.int64))
