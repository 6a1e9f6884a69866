"""Whole chunks of steps in one launch (team kernels) against the separate
kernels of a context with GEMSGPU_NO_TEAM=1 (GPU).

Both run the same per-atom code with the same lanes per atom, so positions,
velocities, forces and list updates agree bit for bit.  FIRE sums its power
over differently sized blocks: its few steps agree to rounding (1e-12 of the
coordinates, about 1e4 roundings of 64-bit arithmetic).
"""
import numpy as np
import pytest

gems = pytest.importorskip("gems_b200")
from gems_b200 import workloads as W  # noqa: E402

pytestmark = pytest.mark.gpu


def lattice(base, a, n, rng, jitter):
    g = np.stack(np.meshgrid(*(np.arange(k) for k in n), indexing="ij"), axis=-1).reshape(-1, 1, 3)
    x = ((g + np.asarray(base)[None]).reshape(-1, 3) + 0.1) * a
    return x + rng.normal(0.0, jitter, x.shape), tuple(k * a for k in n)


FCC = [[0, 0, 0], [.5, .5, 0], [.5, 0, .5], [0, .5, .5]]
DIA = FCC + [[.25, .25, .25], [.75, .75, .25], [.75, .25, .75], [.25, .75, .75]]


def make(ctx, field, geom, prec, integ, lanes, seed, species=1, half=False):
    """One system; geom: cells of a periodic block, or atoms of a cluster."""
    rng = np.random.default_rng(seed)
    L = None
    if field == "lj":
        pos, L = lattice(FCC, (4 / 0.8442) ** (1 / 3), geom, rng, 0.05)
        mass, T, dt = np.ones(len(pos)), 0.72 / W.KB_EV, 0.005 * np.sqrt(W.UI_EV)
    elif field == "tersoff":
        pos, L = lattice(DIA, 5.431, geom, rng, 0.1)
        mass, T, dt = np.full(len(pos), W.MASS["Si"]), 1500.0, 0.001
    else:
        if isinstance(geom, tuple):
            pos, L = lattice(FCC, 4.078, geom, rng, 0.1)
        else:
            pos = W.cluster(geom, rng, check=False)
        mass, T, dt = np.full(len(pos), W.MASS["Au"]), 900.0, 0.004
    typ = (np.arange(len(pos)) % species).astype(np.int32)
    vel = W.maxwell(len(pos), mass, T, rng) if len(pos) > 1 else np.zeros((1, 3))
    s = gems.System(pos, mass, types=typ, ntypes=species, ctx=ctx, vel=vel)
    s.set_box(L, (True, True, True)) if L else s.set_box(None)
    s.set_skin(0.3 if field == "lj" else 0.6)
    if field == "lj":
        s.set_lj(1.0, 1.0, 2.5, eshift=-0.0163)
    elif field == "tersoff":
        s.set_tersoff(W.TERSOFF_SI)
    else:
        for i in range(species):
            for j in range(i, species):
                s.set_smatb(*W.SMATB[("Au", "Pt")[i if i == j else 0]], ti=i, tj=j)
    s.set_half(half)
    s.set_precision(prec)
    s.set_lanes(lanes)
    if integ == "ermak":
        s.set_ermak(dt, 1.0, T, seed=seed)
    elif integ == "vv":
        s.set_vv(dt)
    else:
        s.set_fire(0.002, 0.01)
    return s


def run(monkeypatch, team, build, steps):
    monkeypatch.setenv("GEMSGPU_NO_TEAM", "0" if team else "1")
    ctx = gems.Context()
    try:
        ss = build(ctx)
        n0 = ctx.launches()
        ctx.batch_md_steps(ss, steps)
        launches = ctx.launches() - n0
        return [(s.pos, s.vel, s.acel, s.force, s.epot_atoms, s.nupd) for s in ss], launches
    finally:
        ctx.close()


def same(monkeypatch, build, steps):
    a, la = run(monkeypatch, True, build, steps)
    b, lb = run(monkeypatch, False, build, steps)
    assert la < lb, (la, lb)  # the team launches ran
    for x, y in zip(a, b):
        for u, v in zip(x[:5], y[:5]):
            assert np.isfinite(u).all()
            np.testing.assert_array_equal(u, v)
        assert x[5] == y[5]


# resident form: single atoms and pairs, a cluster of a virtual block more or
# less, the largest, and every number of lanes
@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("n,lanes,steps", [(1, 8, 5), (2, 32, 31), (13, 8, 60), (31, 8, 45), (33, 8, 45), (147, 16, 201),
                                           (147, 1, 40), (309, 2, 40), (640, 4, 60), (500, 32, 20)])
def test_clusters(monkeypatch, prec, n, lanes, steps):
    same(monkeypatch, lambda c: [make(c, "smatb", n, prec, "ermak", lanes, 3)], steps)


# arena form, and both forms with cell lists and odd grids
@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("field,geom,lanes,integ,steps", [
    ("lj", (6, 6, 6), 8, "vv", 61), ("lj", (7, 6, 9), 2, "vv", 60), ("lj", (6, 7, 6), 32, "vv", 33),
    ("lj", (12, 13, 11), 4, "vv", 40), ("smatb", (6, 6, 7), 16, "ermak", 61), ("smatb", (9, 8, 7), 4, "vv", 60),
    ("smatb", (16, 15, 14), 2, "ermak", 40), ("smatb", (5, 5, 5), 1, "vv", 40), ("tersoff", (4, 4, 4), 4, "vv", 61),
    ("tersoff", (6, 5, 7), 4, "vv", 60)])
def test_bulk(monkeypatch, prec, field, geom, lanes, integ, steps):
    same(monkeypatch, lambda c: [make(c, field, geom, prec, integ, lanes, 4)], steps)


@pytest.mark.parametrize("prec", [0, 1])
def test_batches(monkeypatch, prec):
    """Uneven systems side by side, two integrators, alloys, half lists."""
    same(monkeypatch, lambda c: [make(c, "smatb", n, prec, ("vv", "ermak")[n % 2], 4, n, species=2)
                                 for n in (5, 640, 64, 255, 13, 400, 17, 129)], 60)
    same(monkeypatch, lambda c: [make(c, "lj", g, prec, "vv", 4, 7, half=g[0] == 6) for g in ((6, 6, 6), (8, 6, 7))], 60)
    if prec:
        same(monkeypatch, lambda c: [make(c, "tersoff", g, prec, "vv", 2, 7) for g in ((4, 4, 4), (5, 4, 7))], 60)


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("cells", [4, 8])
def test_list_overflow_is_healed(monkeypatch, prec, cells):
    """A dense block in a large box overflows the first list estimate."""
    def build(ctx):
        s = make(ctx, "lj", (cells,) * 3, prec, "vv", 8, 5)
        s.set_box((60.0, 60.0, 60.0), (True, True, True))
        s.set_precision(prec)  # the fixed-point copies follow the new box
        return [s]
    same(monkeypatch, build, 40)


@pytest.mark.parametrize("prec", [0, 1])
@pytest.mark.parametrize("sizes", [(13, 147, 700, 30, 1000), (309,), (1500,)])
def test_fire(monkeypatch, prec, sizes):
    out = []
    for team in (True, False):
        monkeypatch.setenv("GEMSGPU_NO_TEAM", "0" if team else "1")
        ctx = gems.Context()
        ss = [make(ctx, "smatb", n, prec, "fire", 4, 11) for n in sizes]
        it = ctx.batch_fire(ss, 1e-9, 50)
        out.append((it, [s.pos for s in ss], ctx.batch_energy(ss)[0]))
        ctx.close()
    np.testing.assert_array_equal(out[0][0], out[1][0])
    for x, y in zip(out[0][1], out[1][1]):
        np.testing.assert_allclose(x, y, rtol=0, atol=1e-12 * np.abs(y).max())
    np.testing.assert_allclose(out[0][2], out[1][2], rtol=1e-12)


@pytest.mark.parametrize("prec", [0, 1])
def test_pair_functions_over_the_range(prec):
    """A dimer from 1.2 A to beyond the cut-off in steps that meet both
    regimes and their borders, against the oracle.  FP64: 2e-13 of the largest
    value (the exponents reach 10, a rounding of which is 1e-15 relative, and
    the oracle takes other functions); mixed: 4e-6 (single-precision pairs,
    positions on a 2^-22 A grid)."""
    from oracle import oracle as O
    tol = 4e-6 if prec else 2e-13
    for setup in (lambda s: s.set_smatb(*W.SMATB["Au"]), lambda s: s.set_lj(1.0, 2.6, 5.0, eshift=-0.01),
                  lambda s: s.set_lj(1.0, 2.6, 5.0, shifted_force=True)):
        g = gems.System(np.array([[0.0, 0, 0], [3.0, 0, 0]]), W.MASS["Au"])
        o = O.System(np.array([[0.0, 0, 0], [3.0, 0, 0]]), W.MASS["Au"])
        for s in (g, o):
            setup(s)
        g.set_precision(prec)
        e, f, eo, fo = [], [], [], []
        for r in np.concatenate([np.linspace(2.2, 5.2, 40), [4.4, 5.0, np.nextafter(4.4, 0), np.nextafter(5.0, 9)]]):
            x = np.array([[0.1, 0.2, -0.3], [0.1 + r / 3, 0.2 - 2 * r / 3, -0.3 + 2 * r / 3]])
            for s, ee, ff in ((g, e, f), (o, eo, fo)):
                s.set_pos(x)
                ee.append(s.interact())
                ff.append(s.force)
        eo, fo = np.array(eo), np.array(fo)
        ok = np.isfinite(eo) & np.isfinite(fo).all((1, 2))
        if prec:
            ok[[-3, -1]] = False  # r = 5 is the cut-off: on which side is decided by the 2^-22 A grid
        assert np.abs(np.array(e) - eo)[ok].max() <= tol * np.abs(eo[ok]).max()
        assert np.abs(np.array(f) - fo)[ok].max() <= tol * np.abs(fo[ok]).max()


def _noalloc(pos, L, pbc):
    import ctypes
    torch = pytest.importorskip("torch")
    n = len(pos)
    x = torch.tensor(pos.ravel(), dtype=torch.float64, device="cuda")
    f = torch.full((3 * n,), np.nan, dtype=torch.float64, device="cuda")
    e = torch.full((n,), np.nan, dtype=torch.float64, device="cuda")
    L, ip = np.array(L, dtype=float), np.array(pbc, dtype=np.int32)
    rc = gems.lib().gemsgpu_smatb_forces_noalloc(
        ctypes.c_void_p(x.data_ptr()), n, int(ip.any()), L.ctypes.data_as(ctypes.POINTER(ctypes.c_double)),
        ip.ctypes.data_as(ctypes.POINTER(ctypes.c_int)), *W.SMATB["Au"], ctypes.c_void_p(f.data_ptr()),
        ctypes.c_void_p(e.data_ptr()), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    assert rc == 0
    return f.cpu().numpy().reshape(n, 3), e.cpu().numpy()


@pytest.mark.parametrize("k", [0, 70])
def test_noalloc_special_values(k):
    """An atom at infinity (or beyond the squares' range) has no neighbours and
    changes nobody else's forces; a NaN coordinate reaches every atom."""
    pos = W.cluster(147, np.random.default_rng(5), check=False)
    f0, e0 = _noalloc(np.delete(pos, k, 0), [400.0] * 3, [0, 0, 0])
    for far in (np.inf, -np.inf, 1e39, 1e200):
        pos[k] = far
        f, e = _noalloc(pos, [400.0] * 3, [0, 0, 0])
        assert (f[k] == 0.0).all() and e[k] == 0.0
        assert np.abs(np.delete(f, k, 0) - f0).max() <= 1e-12 * np.abs(f0).max()
        assert np.abs(np.delete(e, k) - e0).max() <= 1e-12 * np.abs(e0).max()
    pos[k] = 0.0
    pos[k, 1] = np.nan
    f, e = _noalloc(pos, [400.0] * 3, [0, 0, 0])
    assert np.isnan(f).all() and np.isnan(e).all()


@pytest.mark.parametrize("n,box", [(1, None), (2, None), (31, None), (65, None), (2048, None), (2049, None), (4096, None),
                                   (1372, (28.6, 28.6, 28.6)), (2916, (36.8, 36.8, 36.8)), (2916, (36.8, None, 36.8))])
def test_noalloc_sizes(n, box):
    """gemsgpu_smatb_forces_noalloc at the edges of its tiles and launch shapes,
    clusters off the origin and periodic boxes with atoms outside them, against
    the oracle: 1e-12 of the largest force (sums of 50 terms of 1e-15)."""
    from oracle import oracle as O
    rng = np.random.default_rng(n)
    if box:
        m = round((n / 4) ** (1 / 3))
        pos, _ = lattice(FCC, 4.086, (m, m, m), rng, 0.08)
        pos = pos + np.where(rng.random(pos.shape) < 0.1, 1, 0) * np.array([b or 0.0 for b in box])
    else:
        pos = W.cluster(n, rng, check=False) + np.array([300.0, -40.0, 7.0])
    pbc = [1 if box and b else 0 for b in (box or (0, 0, 0))]
    L = np.array([(b or 400.0) for b in (box or (0, 0, 0))], dtype=float)
    o = O.System(np.mod(pos, np.where(pbc, L, 1e9)) if box else pos, W.MASS["Au"])
    if box:
        o.set_box(L, [bool(p) for p in pbc])
    o.set_skin(0.1)
    o.set_smatb(*W.SMATB["Au"])
    o.interact()
    f, e = _noalloc(pos, L, pbc)
    if n == 1:  # no neighbour: rho = 0, no force
        assert e[0] == 0.0 and (f == 0.0).all()
        return
    assert np.abs(f - o.force).max() <= 1e-12 * np.abs(o.force).max()
    assert np.abs(e - o.epot_atoms).max() <= 1e-12 * np.abs(o.epot_atoms).max()


@pytest.mark.parametrize("n", [63, 64, 65, 129, 240, 256, 257, 300])
def test_crowded_cells(n):
    """A cell of n atoms (every one within a cut-off of the others), at the
    edges of the cell sort's paths: the pairs are all pairs within the list
    cut-off, in the oracle's order where its rows (256 entries) hold them."""
    from oracle import oracle as O
    rng = np.random.default_rng(n)
    pos = np.concatenate([rng.uniform(10.5, 13.5, (n, 3)), rng.uniform(0.0, 64.0, (1000, 3))])
    s = gems.System(pos, np.ones(len(pos)))
    s.set_box((64.0,) * 3, (True,) * 3)
    s.set_skin(0.3)
    s.set_lj(1.0, 0.05, 5.3)
    s.interact()
    d = pos[:, None] - pos[None]
    d -= 64.0 * np.rint(d / 64.0)
    near = (d ** 2).sum(-1) < 5.6 ** 2
    np.fill_diagonal(near, False)
    i, j = np.nonzero(near)
    assert np.array_equal(s.pair_set(), i * len(pos) + j)
    if n <= 240:
        o = O.System(pos, np.ones(len(pos)))
        o.set_box((64.0,) * 3, (True,) * 3)
        o.set_skin(0.3)
        o.set_lj(1.0, 0.05, 5.3)
        o.interact()
        (nn, a), (mm, b) = s.neighbour_list(), o.neighbour_list()
        assert np.array_equal(nn, mm)
        assert all(np.array_equal(a[:c, k], b[:c, k]) for k, c in enumerate(nn))


@pytest.mark.parametrize("cells,pbc", [((14, 14, 13), (True, True, True)), ((16, 16, 16), (True, False, True)),
                                       ((21, 21, 21), (True, True, True)), ((6, 30, 20), (True, True, False)),
                                       ((6, 30, 20), (True, True, True))])
def test_sparse_force_lists(cells, pbc):
    """Force lists of sparse cells (one thread, three or nine per atom; three
    cells a side; open faces): forces equal the oracle's, on the first list and
    on one built after every atom has moved, and the list is the oracle's then.
    1e-11 of the largest force: sums of 100 terms of 1e-16 and their
    cancellation."""
    from oracle import oracle as O
    rng = np.random.default_rng(sum(cells))
    g = np.stack(np.meshgrid(*[np.arange(c) for c in cells], indexing="ij"), -1).reshape(-1, 3)
    L = tuple(1.6 * c for c in cells)
    pos = (g + 0.5) * 1.6 + rng.uniform(-0.15, 0.15, g.shape)
    o, s = O.System(pos, np.ones(len(pos))), gems.System(pos, np.ones(len(pos)))
    for q in (o, s):
        q.set_box(L, pbc)
        q.set_skin(0.3)
        q.set_lj(1.0, 1.0, 2.5)
    for shift in (0.0, 0.25):
        x = pos + np.where(rng.random(pos.shape) < 0.5, shift, -shift)
        o.set_pos(x)
        s.set_pos(x)
        o.interact()
        s.interact()
        assert np.abs(s.force - o.force).max() <= 1e-11 * np.abs(o.force).max()
        (nn, a), (mm, b) = s.neighbour_list(), o.neighbour_list()
        assert np.array_equal(nn, mm)
        assert all(np.array_equal(a[:c, k], b[:c, k]) for k, c in enumerate(nn))
