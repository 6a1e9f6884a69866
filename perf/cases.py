"""The work that users of the library have it do, as timed cases.

A case is a dict of plain values: what is called (`kind`), the force field,
the geometry, the precision, the integrator and the number of steps.  Every
pass goes through the Python binding of the C ABI, from host arrays to host
arrays, as a program that owns its trajectory does.

kinds
  forces   a caller that keeps its own integrator: new positions in, one
           force evaluation, energies and forces out, every step
  noalloc  the same for a caller with its own device buffers
           (gemsgpu_smatb_forces_noalloc)
  md       set the state, run a block of steps on the device, read it back
  npt      the next block of a run under the G-JF piston, with the box and the
           virial
  fire     relax a batch of free clusters for a fixed number of iterations

Results of mixed-precision systems come back as single precision: that is
what their users keep (frames, training data), and all the pair math holds.
"""
import ctypes
import math

import numpy as np
import torch

import gems_b200 as gems
from gems_b200 import workloads as W

# ---- the listed cases

A_AU, A_SI = 4.078, 5.431
A_LJ = (4.0 / 0.8442) ** (1.0 / 3.0)


def listed():
    return [
        # one evaluation of a 147-atom cluster per step of somebody else's
        # integrator or minimiser: launches and latency
        _case("forces_au147_fp64", "forces", "smatb", n=147, prec="fp64"),
        # the same drop-in call at the size of a production crystal
        _case("forces_au32k_mixed", "forces", "smatb", nx=20, ny=20, nz=20, prec="mixed"),
        # a host program with a fixed device-memory budget
        _case("noalloc_au4000_fp64", "noalloc", "smatb", nx=10, ny=10, nz=10, prec="fp64"),
        # 64 replicas of a 147-atom cluster between two exchange rounds
        _case("replicas_64xau147_mixed", "md", "smatb", n=147, count=64, prec="mixed", integ="ermak", temp=300.0,
              steps=100),
        # the 4000-atom Lennard-Jones fluid in the precision of the Fortran program
        _case("md_lj4000_fp64", "md", "lj", nx=10, ny=10, nz=10, prec="fp64", temp=0.72, steps=100),
        # sixteen such fluids together (a parameter sweep)
        _case("md_16xlj4000_mixed", "md", "lj", nx=10, ny=10, nz=10, count=16, prec="mixed", temp=0.72, steps=100),
        # a Langevin run of the 32000-atom gold crystal, FP64 throughout
        _case("md_au32k_fp64", "md", "smatb", nx=20, ny=20, nz=20, prec="fp64", integ="ermak", temp=300.0, steps=100),
        # eight replicas of it in mixed precision: the throughput workload
        _case("md_8xau32k_mixed", "md", "smatb", nx=20, ny=20, nz=20, count=8, prec="mixed", integ="ermak",
              temp=300.0, steps=100),
        # the crystal at constant pressure, which needs the virial each step
        _case("npt_au32k_mixed", "npt", "smatb", nx=20, ny=20, nz=20, prec="mixed", temp=300.0, steps=50),
        # bond-order silicon: the accuracy reference, and the largest crystal
        _case("md_si32k_fp64", "md", "tersoff", nx=16, ny=16, nz=16, prec="fp64", temp=1000.0, steps=50),
        _case("md_si1M_mixed", "md", "tersoff", nx=50, ny=50, nz=50, prec="mixed", temp=1000.0, steps=50),
        # relaxing a set of free clusters of 13 to 2000 atoms
        _case("fire_128_clusters_mixed", "fire", "smatb", n=2000, count=128, prec="mixed", steps=100),
    ]


def _case(name, kind, field, n=0, nx=0, ny=0, nz=0, count=1, prec="fp64", integ="vv", temp=300.0, steps=1, species=1):
    c = dict(kind=kind, field=field, n=n, nx=nx, ny=ny, nz=nz, count=count, prec=prec, integ=integ, temp=temp,
             steps=steps, species=species)
    if name:
        c["name"] = name
    return c


# ---- drawn cases: the same ranges, odd sizes and uneven boxes among them

def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _cells(rng, lo, hi, per):
    """An uneven block of unit cells holding lo..hi atoms, `per` a cell."""
    n = _log(rng, lo, hi) / per
    a, b = (math.exp(rng.uniform(-0.25, 0.25)) for _ in range(2))
    e = n ** (1.0 / 3.0)
    return [max(6, int(round(e * f))) for f in (a, b, 1.0 / (a * b))]  # three list cut-offs or more


def draw(rng):
    prec = rng.choice(("fp64", "mixed"))
    what = rng.choice(("cluster_forces", "bulk_forces", "noalloc", "replicas", "lj", "au", "npt", "si", "fire"))
    species = rng.choice((1, 1, 2))
    if what == "cluster_forces":
        return _case(None, "forces", "smatb", n=_log(rng, 13, 5000), prec=prec, species=species)
    if what == "bulk_forces":
        x, y, z = _cells(rng, 500, 100000, 4)
        return _case(None, "forces", "smatb", nx=x, ny=y, nz=z, prec=prec, species=species)
    if what == "noalloc":
        if rng.random() < 0.5:
            return _case(None, "noalloc", "smatb", n=_log(rng, 13, 5000))
        x, y, z = _cells(rng, 300, 12000, 4)
        return _case(None, "noalloc", "smatb", nx=x, ny=y, nz=z)
    if what == "replicas":
        return _case(None, "md", "smatb", n=_log(rng, 13, 2000), count=_log(rng, 1, 64), prec=prec,
                     integ=rng.choice(("vv", "ermak")), temp=rng.uniform(200.0, 600.0), steps=rng.randint(20, 100),
                     species=species)
    if what == "lj":
        x, y, z = _cells(rng, 400, 60000, 4)
        return _case(None, "md", "lj", nx=x, ny=y, nz=z, count=_log(rng, 1, 8), prec=prec,
                     temp=rng.uniform(0.5, 0.9), steps=rng.randint(20, 100))
    if what == "au":
        x, y, z = _cells(rng, 1000, 60000, 4)
        return _case(None, "md", "smatb", nx=x, ny=y, nz=z, count=_log(rng, 1, 8), prec=prec,
                     integ=rng.choice(("vv", "ermak")), temp=rng.uniform(200.0, 600.0), steps=rng.randint(20, 80),
                     species=species)
    if what == "npt":
        x, y, z = _cells(rng, 2500, 60000, 4)
        x, y, z = max(x, 7), max(y, 7), max(z, 7)  # a moving box keeps four cells or more
        return _case(None, "npt", "smatb", nx=x, ny=y, nz=z, prec=prec, temp=rng.uniform(200.0, 500.0),
                     steps=rng.randint(20, 50))
    if what == "si":
        x, y, z = _cells(rng, 1000, 400000, 8)
        return _case(None, "md", "tersoff", nx=x, ny=y, nz=z, prec=prec, temp=rng.uniform(300.0, 1200.0),
                     steps=rng.randint(10, 50))
    return _case(None, "fire", "smatb", n=_log(rng, 100, 2000), count=_log(rng, 1, 128), prec=prec,
                 steps=50 * rng.randint(1, 2), species=species)


# ---- inputs, from the seed alone

def _block(base, a, nx, ny, nz):
    """nx x ny x nz unit cells, set a quarter spacing off the box faces."""
    g = np.stack(np.meshgrid(np.arange(nz), np.arange(ny), np.arange(nx), indexing="ij")[::-1], axis=-1)
    pos = (g.reshape(-1, 1, 3) + np.asarray(base)[None]).reshape(-1, 3) * a
    return pos, (nx * a, ny * a, nz * a)


_FCC = [[0.25, 0.25, 0.25], [0.75, 0.75, 0.25], [0.75, 0.25, 0.75], [0.25, 0.75, 0.75]]
_DIA = [[x + s, y + s, z + s] for s in (0.125, 0.375) for x, y, z in ((0, 0, 0), (.5, .5, 0), (.5, 0, .5), (0, .5, .5))]
_ELEMENTS = ("Au", "Pt")  # one species, or gold with a quarter of platinum
_MIX = tuple(0.5 * (a + b) for a, b in zip(W.SMATB["Au"], W.SMATB["Pt"]))


def _cluster_sizes(case):
    """`count` sizes spread evenly over the logarithm of 13..n."""
    k = case["count"]
    return [int(round(13.0 * (case["n"] / 13.0) ** ((i + 0.5) / k))) for i in range(k)]


def _inputs(case, seed):
    """A list of systems: pos, vel, type, mass, L (None: a free cluster)."""
    rng = np.random.default_rng([seed, 20240611])
    field, out = case["field"], []
    sizes = [case["n"]] * case["count"]
    if case["kind"] == "fire":
        sizes = _cluster_sizes(case)
    for n in sizes:
        L, kT = None, case["temp"]
        if field == "lj":  # displaced lattice of the fluid's density: it melts as it runs
            pos, L = _block(_FCC, A_LJ, case["nx"], case["ny"], case["nz"])
            pos = pos + rng.normal(0.0, 0.05, pos.shape)
            kT = case["temp"] / W.KB_EV
        elif field == "tersoff":  # thermal displacements of the crystal
            pos, L = _block(_DIA, A_SI, case["nx"], case["ny"], case["nz"])
            pos = pos + rng.normal(0.0, 0.1 * math.sqrt(case["temp"] / 1000.0), pos.shape)
        elif case["nx"]:
            pos, L = _block(_FCC, A_AU, case["nx"], case["ny"], case["nz"])
            pos = pos + rng.normal(0.0, 0.085 * math.sqrt(case["temp"] / 300.0), pos.shape)
        else:
            pos = W.cluster(n, rng, check=False)
        m = len(pos)
        typ = (rng.random(m) < 0.25).astype(np.int32) if case["species"] == 2 else np.zeros(m, dtype=np.int32)
        if field == "lj":
            mass = np.ones(m)
        elif field == "tersoff":
            mass = np.full(m, W.MASS["Si"])
        else:
            mass = np.array([W.MASS[e] for e in _ELEMENTS])[typ]
        vel = np.zeros((m, 3)) if case["kind"] == "fire" else W.maxwell(m, mass, kT, rng)
        out.append(dict(pos=np.ascontiguousarray(pos), vel=np.ascontiguousarray(vel), type=typ, mass=mass, L=L))
    return out


def _dt(case):
    return {"lj": 0.005 * math.sqrt(W.UI_EV), "tersoff": 0.001, "smatb": 0.002}[case["field"]]


_LJ_RC = 2.5
_LJ_SHIFT = 4.0 * ((1.0 / _LJ_RC) ** 12 - (1.0 / _LJ_RC) ** 6)


def _setup(s, case, w, k):
    s.set_box(w["L"], (True, True, True)) if w["L"] else s.set_box(None)
    s.set_skin(0.3 if case["field"] == "lj" else 1.0)
    if case["field"] == "lj":
        s.set_lj(1.0, 1.0, _LJ_RC, eshift=_LJ_SHIFT)
    elif case["field"] == "tersoff":
        s.set_tersoff(W.TERSOFF_SI)
    else:
        s.set_smatb(*W.SMATB["Au"])
        if case["species"] == 2:
            s.set_smatb(*W.SMATB["Pt"], ti=1, tj=1)
            s.set_smatb(*_MIX, ti=0, tj=1)
    s.set_precision(gems.PREC_MIXED if case["prec"] == "mixed" else gems.PREC_FP64)
    if case["kind"] == "md":
        if case["integ"] == "ermak":
            s.set_ermak(_dt(case), 1.0, case["temp"], seed=1000 + k)
        else:
            s.set_vv(_dt(case))
    elif case["kind"] == "npt":
        s.set_lgf(_dt(case), case["temp"], 1.0, 1.0, 1.0, 1e-3, seed=1000 + k)
    elif case["kind"] == "fire":
        s.set_fire(0.002, 0.01)


def _host(n):
    """A pinned host buffer, which a program that copies every block keeps."""
    return torch.empty((n, 3), dtype=torch.float64, pin_memory=torch.cuda.is_available()).numpy()


def _pinned(a):
    b = _host(len(a))
    b[:] = a
    return b


def prepare(case, seed):
    ws = _inputs(case, seed)
    if case["kind"] == "noalloc":
        w = ws[0]
        dev = torch.device("cuda", 0)
        n = len(w["pos"])
        L = np.ascontiguousarray(w["L"] or (0.0, 0.0, 0.0), dtype=np.float64)
        return dict(case=case, n=n, x=torch.tensor(w["pos"].ravel(), dtype=torch.float64, device=dev),
                    f=torch.empty(3 * n, dtype=torch.float64, device=dev),
                    e=torch.empty(n, dtype=torch.float64, device=dev), boxed=1 if w["L"] else 0, L=L,
                    pbc=np.full(3, 1 if w["L"] else 0, dtype=np.int32), fn=gems.lib().gemsgpu_smatb_forces_noalloc)
    ctx = gems.Context(max_atoms=sum(len(w["pos"]) for w in ws), max_systems=len(ws) + 1)
    ss = []
    for k, w in enumerate(ws):
        s = gems.System(w["pos"], w["mass"], types=w["type"], ntypes=case["species"], ctx=ctx, vel=w["vel"])
        _setup(s, case, w, k)
        ss.append(s)
    state = dict(case=case, ctx=ctx, ss=ss)
    if case["kind"] == "fire":
        for s in ss:
            s.set_lanes(4, 1)
    else:
        ctx.batch_autotune(ss, 10)
    if case["kind"] == "forces":
        # two frames of the caller's trajectory, taken in turn
        rng = np.random.default_rng([seed, 7])
        x = ws[0]["pos"]
        state.update(frames=[np.ascontiguousarray(x), np.ascontiguousarray(x + rng.normal(0.0, 0.01, x.shape))], turn=0)
    else:
        state.update(pos=[_pinned(w["pos"]) for w in ws], vel=[_pinned(w["vel"]) for w in ws],
                     pos_out=[_host(s.n) for s in ss], vel_out=[_host(s.n) for s in ss])
    return state


# ---- one pass

def _kept(case, a):
    """What a user keeps of a result: mixed-precision results as float32."""
    t = torch.from_numpy(a) if isinstance(a, np.ndarray) else torch.tensor(a, dtype=torch.float64)
    return t.to(torch.float32) if case["prec"] == "mixed" else t


def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "noalloc":
        rc = state["fn"](_ptr(state["x"]), state["n"], state["boxed"],
                         state["L"].ctypes.data_as(ctypes.POINTER(ctypes.c_double)),
                         state["pbc"].ctypes.data_as(ctypes.POINTER(ctypes.c_int)), *W.SMATB["Au"],
                         _ptr(state["f"]), _ptr(state["e"]),
                         ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        if rc != 0:
            raise RuntimeError("gemsgpu_smatb_forces_noalloc: %d" % rc)
        return {"force": state["f"], "epot_atoms": state["e"]}
    ss, ctx = state["ss"], state["ctx"]
    if kind == "forces":
        s = ss[0]
        s.set_pos(state["frames"][state["turn"] % 2])
        state["turn"] += 1
        e = s.interact()
        return {"epot": _kept(case, e), "force": _kept(case, s.force)}
    out = {}
    if kind != "npt":  # the run at constant pressure goes on from block to block
        ctx.batch_set_state(ss, state["pos"], state["vel"])
    if kind == "fire":
        for s in ss:
            s.set_fire(0.002, 0.01)
        out["iters"] = ctx.batch_fire(ss, 1e-7, case["steps"])  # never reached: a fixed number of iterations
        ep, _, _ = ctx.batch_get_state(ss, state["pos_out"], None)
        out["epot"] = _kept(case, ep)
    else:
        ctx.batch_md_steps(ss, case["steps"])
        ep, ek, t = ctx.batch_get_state(ss, state["pos_out"], state["vel_out"])
        out["epot"], out["ekin"], out["temp"] = (_kept(case, v) for v in (ep, ek, t))
        out["vel"] = _whole(case, state["vel_out"])
        if kind == "npt":
            out["box"], out["virial"] = _kept(case, ss[0].box_now()), _kept(case, ss[0].virial_ev())
    out["pos"] = _whole(case, state["pos_out"])
    return out


def _whole(case, arrays):
    """One array of all systems' atoms."""
    t = [torch.from_numpy(a) for a in arrays]
    if case["prec"] == "mixed":
        out = torch.empty((sum(len(a) for a in t), 3), dtype=torch.float32)
        o = 0
        for a in t:
            out[o:o + len(a)].copy_(a)
            o += len(a)
        return out
    return t[0] if len(t) == 1 else torch.cat(t)


# ---- what a pass cannot do without

def work(case):
    if case["kind"] == "fire":
        n = sum(_cluster_sizes(case))
    else:
        per = case["nx"] * case["ny"] * case["nz"] * (8 if case["field"] == "tersoff" else 4)
        n = case["count"] * (per or case["n"])
    # flops of an evaluation: half the atoms within the cut-off, each pair
    # once (density and force 60, Lennard-Jones 25), or bonds and triplets
    flops = {"smatb": 21 * 60, "lj": 27.6 * 25, "tersoff": 660}[case["field"]]
    if case["kind"] in ("forces", "noalloc"):
        return {"bytes": 56.0 * n, "flops": float(flops * n)}
    # positions and velocities in and out once; per step the forces and 30
    # flops of the integrator
    return {"bytes": 96.0 * n, "flops": float((flops + 30) * n * case["steps"])}


# ---- the same in plain FP64 torch

_EV_UI = 1.0 / (1.0e4 * 1.6605402e-27 / 1.60219e-19)
_KB_EV = 8.617385e-05


def exact(case, seed):
    if case["kind"] == "npt" or case["integ"] == "ermak":
        return None  # their noise is the library's own random stream
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    ws = _inputs(case, seed)
    x = torch.tensor(np.concatenate([w["pos"] for w in ws]), device=dev)
    v = torch.tensor(np.concatenate([w["vel"] for w in ws]), device=dev)
    m = torch.tensor(np.concatenate([w["mass"] for w in ws]), device=dev)[:, None]
    typ = torch.tensor(np.concatenate([w["type"] for w in ws]), device=dev).long()
    own = torch.repeat_interleave(torch.arange(len(ws), device=dev), torch.tensor([len(w["pos"]) for w in ws], device=dev))
    L = torch.tensor(ws[0]["L"], dtype=torch.float64, device=dev) if ws[0]["L"] else None
    field = {"lj": _lj, "tersoff": _tersoff, "smatb": _smatb}[case["field"]]
    rcut = {"lj": _LJ_RC, "tersoff": W.TERSOFF_SI[9] + W.TERSOFF_SI[10], "smatb": max(W.SMATB["Au"][6], W.SMATB["Pt"][6])}[
        case["field"]]
    keep = 0.6 if case["field"] == "lj" else 1.5
    lists = {}

    def forces(x):
        if "x" not in lists or float((x - lists["x"]).norm(dim=1).max()) > 0.5 * keep:
            lists["x"], lists["ij"] = x.clone(), _pairs(x, own, L, rcut + keep)
        i, j = lists["ij"]
        y = x.detach().requires_grad_(True)
        d = y[j] - y[i]
        if L is not None:
            d = d - L * torch.round(d.detach() / L)
        e = field(d, i, j, typ, len(x))
        (g,) = torch.autograd.grad(e.sum(), y)
        return e.detach() * _EV_UI, -g * _EV_UI

    def total(e):
        return torch.zeros(len(ws), dtype=torch.float64, device=dev).index_add_(0, own, e)

    if case["kind"] in ("forces", "noalloc"):
        e, f = forces(x)
        if case["kind"] == "noalloc":
            return {"force": f.reshape(-1).cpu(), "epot_atoms": e.cpu()}
        return {"epot": e.sum().cpu(), "force": f.cpu()}
    wrapped = (lambda y: y - L * torch.floor(y / L)) if L is not None else (lambda y: y)
    e, f = forces(x)
    dt = torch.full((len(ws), 1), 0.002 if case["kind"] == "fire" else _dt(case), dtype=torch.float64, device=dev)
    alpha, npos = torch.full_like(dt, 0.1), torch.zeros_like(dt)
    for _ in range(case["steps"]):
        h = dt[own]
        v = v + 0.5 * h * f / m
        x = x + h * v
        e, f = forces(x)
        v = v + 0.5 * h * f / m
        if case["kind"] == "fire":
            p = total((v * f).sum(1))[:, None]
            a = alpha[own]
            v = (1 - a) * v + a * v.norm(dim=1, keepdim=True) * f / f.norm(dim=1, keepdim=True)
            up = p > 0
            npos = torch.where(up, npos + 1, torch.zeros_like(npos))
            fast = up & (npos > 5)
            dt = torch.where(fast, (1.1 * dt).clamp(max=0.01), torch.where(up, dt, 0.5 * dt))
            alpha = torch.where(fast, 0.99 * alpha, torch.where(up, alpha, torch.full_like(alpha, 0.1)))
            v = torch.where(up[own], v, torch.zeros_like(v))
    ep = total(e) / _EV_UI
    if case["kind"] == "fire":
        return {"iters": None, "epot": ep.cpu(), "pos": x.cpu()}
    n = torch.bincount(own).double()
    mt = total(m[:, 0])
    vcm = torch.stack([total(m[:, 0] * v[:, k]) for k in range(3)], dim=1) / mt[:, None]
    ek = 0.5 * total((m * (v - vcm[own]) ** 2).sum(1)) / _EV_UI
    return {"epot": ep.cpu(), "ekin": ek.cpu(), "temp": (2.0 * ek / (_KB_EV * 3.0 * n)).cpu(), "vel": v.cpu(),
            "pos": wrapped(x).cpu()}


def _pairs(x, own, L, rc):
    """All ordered pairs of one system closer than rc, sorted by the first."""
    n = len(x)
    if L is not None and n > 20000 and own[-1] == 0 and bool((L / rc >= 3).all()):
        return _pairs_grid(x, L, rc)
    ii, jj = [], []
    starts = torch.bincount(own).cumsum(0)
    lo = 0
    for hi in starts.tolist():
        y = x[lo:hi]
        step = max(1, int(3e7 // len(y)))
        for a in range(0, len(y), step):
            d = y[a:a + step, None, :] - y[None, :, :]
            if L is not None:
                d = d - L * torch.round(d / L)
            i, j = torch.nonzero((d * d).sum(2) < rc * rc, as_tuple=True)
            i = i + a
            ii.append(i[i != j] + lo)
            jj.append(j[i != j] + lo)
        lo = hi
    return torch.cat(ii), torch.cat(jj)


def _pairs_grid(x, L, rc):
    nc = torch.floor(L / rc).long()
    c = torch.minimum((torch.remainder(x, L) / L * nc).long(), nc - 1)
    cid = (c[:, 0] * nc[1] + c[:, 1]) * nc[2] + c[:, 2]
    ncell = int(nc.prod())
    order = torch.argsort(cid)
    cnt = torch.bincount(cid, minlength=ncell)
    beg = cnt.cumsum(0) - cnt
    slot = torch.arange(int(cnt.max()), device=x.device)
    ii, jj = [], []
    for dx in (-1, 0, 1):
        for dy in (-1, 0, 1):
            for dz in (-1, 0, 1):
                q = torch.remainder(c + torch.tensor([dx, dy, dz], device=x.device), nc)
                q = (q[:, 0] * nc[1] + q[:, 1]) * nc[2] + q[:, 2]
                i, k = torch.nonzero(slot[None, :] < cnt[q][:, None], as_tuple=True)
                j = order[beg[q[i]] + k]
                d = x[j] - x[i]
                d = d - L * torch.round(d / L)
                ok = ((d * d).sum(1) < rc * rc) & (i != j)
                ii.append(i[ok])
                jj.append(j[ok])
    i, j = torch.cat(ii), torch.cat(jj)
    o = torch.argsort(i, stable=True)
    return i[o], j[o]


def _lj(d, i, j, typ, n):
    r2 = (d * d).sum(1)
    s6 = 1.0 / r2 ** 3
    p = torch.where(r2 <= _LJ_RC ** 2, 4.0 * (s6 * s6 - s6) - _LJ_SHIFT, torch.zeros_like(r2))
    return torch.zeros(n, dtype=torch.float64, device=d.device).index_add(0, i, 0.5 * p)


def _tail(f, a, rci, rce, r0):
    """The quintic without its first three terms that continues f exp(-a (r/r0 - 1))
    with its first two derivatives from rci to zero at rce."""
    t = rci - rce
    y = f * math.exp(-a * (rci / r0 - 1.0))
    M = np.array([[t ** 5, t ** 4, t ** 3], [5 * t ** 4, 4 * t ** 3, 3 * t ** 2], [20 * t ** 3, 12 * t ** 2, 6 * t]])
    return np.linalg.solve(M, np.array([y, -a / r0 * y, (a / r0) ** 2 * y]))


def _smatb(d, i, j, typ, n):
    rows = [W.SMATB["Au"], _MIX, W.SMATB["Pt"]]
    tab = []
    for A, xi, p, q, r0, rci, rce in rows:
        tab.append([A, xi, p, q, r0, rci, rce, *_tail(xi, q, rci, rce, r0), *_tail(A, p, rci, rce, r0)])
    A, xi, p, q, r0, rci, rce, b1, b2, b3, r1, r2, r3 = torch.tensor(tab, dtype=torch.float64, device=d.device)[
        typ[i] + typ[j]].unbind(1)
    r = (d * d).sum(1).sqrt()
    t = r - rce
    inner, live = r <= rci, r <= rce
    band = torch.where(inner, xi * torch.exp(-q * (r / r0 - 1.0)), ((b1 * t + b2) * t + b3) * t ** 3)
    rep = torch.where(inner, A * torch.exp(-p * (r / r0 - 1.0)), ((r1 * t + r2) * t + r3) * t ** 3)
    zero = torch.zeros_like(r)
    z = torch.zeros(n, dtype=torch.float64, device=d.device)
    rho = z.index_add(0, i, torch.where(live, band * band, zero))
    return z.index_add(0, i, torch.where(live, rep, zero)) - rho.sqrt()


def _tersoff(d, i, j, typ, n):
    A, B, l1, l2, beta, en, c, dd, h, R, D, chi = W.TERSOFF_SI
    with torch.no_grad():
        near = torch.nonzero((d * d).sum(1) <= (R + D) ** 2)[:, 0]
    d, i = d[near], i[near]
    cnt = torch.bincount(i, minlength=n)
    beg = cnt.cumsum(0) - cnt
    k = torch.arange(len(i), device=d.device) - beg[i]
    mb = int(cnt.max())
    r = (d * d).sum(1).sqrt()
    u = torch.zeros(n, mb, 3, dtype=torch.float64, device=d.device).index_put((i, k), d / r[:, None])
    r = torch.ones(n, mb, dtype=torch.float64, device=d.device).index_put((i, k), r)
    on = torch.arange(mb, device=d.device)[None, :] < cnt[:, None]
    fc = torch.where(r < R - D, torch.ones_like(r), 0.5 - 0.5 * torch.sin(0.5 * math.pi * (r - R) / D)) * on
    cos = u @ u.transpose(1, 2)
    g = 1.0 + (c / dd) ** 2 - c * c / (dd * dd + (h - cos) ** 2)
    g = g * (1.0 - torch.eye(mb, dtype=torch.float64, device=d.device))
    zeta = (g * fc[:, None, :]).sum(2)
    some = zeta > 1e-15
    x = (beta * torch.where(some, zeta, torch.ones_like(zeta))) ** en
    b = torch.where(some, chi * (1.0 + x) ** (-0.5 / en), torch.full_like(zeta, chi))
    return (0.5 * fc * (A * torch.exp(-l1 * r) - b * B * torch.exp(-l2 * r))).sum(1)
