"""Performance cases of the package: what a simulation program has it do, through the Python API
(``pdcuda``) and the C ABI under it.

Every case is a body on a (possibly jittered) lattice, the discretisation that ``uniform_box``
makes, with one of the materials, and one pass of one of the solvers over it:

  vv        the body is put into a state, advances a block of Velocity Verlet steps and its fields
            are read: the export interval of a job, or a restart
  relax     a dynamic relaxation from the unloaded state
  newton    one load increment of the quasi-static Newton-Krylov solver from the unloaded state
  ensemble  independent specimens of different sizes, each on its own stable step, together
  static    one force evaluation on arrays that the caller owns on the device

FP64 is the package's default precision and runs in its default lane mapping (one point per
thread, no autotuning). The FP32-compensated form is what a long run of a large body is tuned
for: its cases of 100,000 points and more pin the mapping that the autotuner settles on for such
bodies (one point per thread, 128 threads, packed kernels) so that every run takes the same one,
and launch their steps as CUDA graphs; smaller ones keep the defaults. The FP32 form's fields are
handed on as float32, the precision of its bond arithmetic.

Loads: the outermost layers are pulled apart at a constant speed, on top of a smooth initial
velocity field that the seed draws (and, for jittered bodies, the lattice noise).
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "peridynamics.jl_b200"))
import pdcuda as pd  # noqa: E402
from pdcuda import _lib as L  # noqa: E402
from pdcuda import dynamic_relaxation as drm  # noqa: E402
from pdcuda import newton_krylov as nkm  # noqa: E402

DX = 1e-3
RHO, YOUNG, NU, GC = 2700.0, 70e9, 0.25, 100.0
SAFETY = 0.7
STATIC_MAX = 1 << 18


def listed():
    return [
        # the smallest calls, where latency counts: the mode-I plate with its edge crack (3,200
        # points, bond-based), as a user who only asked for CUDA graphs runs it
        dict(name="plate_bb_f64", kind="vv", nx=40, ny=20, nz=4, mat="BB", prec="fp64", steps=200,
             graph=50, crack=True, tear=True),
        # a coupon of under a thousand points in the FP32 form, eager launches, nothing tuned
        dict(name="coupon_osb_f32", kind="vv", nx=25, ny=13, nz=3, mat="OSB", prec="fp32", steps=60,
             graph=0, crack=True),
        # correspondence in the defaults (FP64, Saint Venant-Kirchhoff), a ragged block
        dict(name="block_cmat_f64", kind="vv", nx=41, ny=29, nz=23, mat="C", model="svk",
             prec="fp64", steps=20, graph=0),
        # ordinary state-based in the defaults, an ordinary size
        dict(name="block_osb_f64", kind="vv", nx=100, ny=50, nz=25, mat="OSB", prec="fp64", steps=20,
             graph=0),
        # bond-based in the defaults at a size where FP64 is still affordable
        dict(name="block_bb_f64", kind="vv", nx=121, ny=67, nz=49, mat="BB", prec="fp64", steps=20,
             graph=0),
        # one million points bond-based, tuned
        dict(name="block_bb_f32", kind="vv", nx=200, ny=100, nz=50, mat="BB", prec="fp32", steps=40,
             graph=20),
        # an ensemble of correspondence specimens (neo-Hooke) of 15,000 to 150,000 points
        dict(name="ensemble_cmat_f32", kind="ensemble", specimens=6, nx=18, mat="C",
             model="neohooke", prec="fp32", steps=40, graph=20, classes=2),
        # the jittered million-point block: no two bonds alike
        dict(name="jitter_osb_f32", kind="vv", nx=200, ny=100, nz=50, mat="OSB", prec="fp32",
             steps=40, graph=20, jitter=0.05),
        # the largest: four million points, ragged
        dict(name="large_osb_f32", kind="vv", nx=211, ny=199, nz=101, mat="OSB", prec="fp32",
             steps=40, graph=20),
        # dynamic relaxation of a bar in tension, the defaults
        dict(name="relax_osb_f64", kind="relax", nx=80, ny=40, nz=20, mat="OSB", prec="fp64",
             steps=40),
        # quasi-static bending of a bond-based beam, one of twenty load increments
        dict(name="newton_beam_f64", kind="newton", nx=60, ny=12, nz=10, mat="BB", prec="fp64"),
        # force evaluations for a host that owns the device memory
        dict(name="static_osb_f64", kind="static", nx=43, ny=31, nz=23, mat="OSB", prec="fp64"),
    ]


def draw(rng):
    """Another case of the same ranges: any solver, material, precision and size between a few
    hundred and a few million points, odd sizes among them."""
    kind = rng.choices(("vv", "relax", "ensemble", "static", "newton"), (12, 2, 2, 2, 1))[0]
    if kind == "newton":
        ny, nz = rng.randint(7, 13), rng.randint(6, 11)
        return dict(kind=kind, nx=rng.randint(40, 70), ny=ny, nz=nz, mat="BB", prec="fp64")
    if kind == "static":
        nx, ny, nz = _box(rng, 500, 200_000)
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, mat="OSB", prec="fp64",
                    jitter=rng.choice((0.0, 0.05)))
    if kind == "ensemble":
        return dict(kind=kind, specimens=rng.randint(3, 7), nx=rng.randint(7, 14), mat="C",
                    model="neohooke", prec="fp32", steps=40, graph=20, classes=rng.randint(1, 3))
    mat = rng.choice(("BB", "OSB", "OSB", "C"))
    prec = rng.choice(("fp64", "fp32"))
    if kind == "relax":
        nx, ny, nz = _box(rng, 2_000, 150_000)
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, mat=rng.choice(("BB", "OSB")), prec="fp64",
                    steps=rng.randint(20, 60))
    nx, ny, nz = _box(rng, 800, 4_000_000 if prec == "fp32" else 600_000 if mat != "C" else 150_000)
    n = nx * ny * nz
    c = dict(kind=kind, nx=nx, ny=ny, nz=nz, mat=mat, prec=prec,
             steps=40 if n > 20_000 else rng.choice((40, 60, 120)))
    if prec == "fp64" and n > 20_000:
        c["steps"] = 20
    c["graph"] = 20 if (prec == "fp32" and n >= 100_000) else rng.choice((0, 20))
    c["jitter"] = rng.choice((0.0, 0.0, 0.05))
    if mat == "C":
        c["model"] = rng.choice(("svk", "neohooke"))
        c["zem"] = rng.choice(("silling", "silling", "wan"))
    if mat == "OSB":
        c["kernel"] = rng.choice(("linear", "linear", "linear", "cubic"))
    if n < 300_000:
        c["m"] = rng.choice((3.015, 3.015, 2.015, 4.015))
    c["crack"] = mat != "C" and rng.random() < 0.3
    return c


def _box(rng, lo, hi):
    n = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    a, b = rng.uniform(1.0, 2.5), rng.uniform(1.0, 3.0)
    nz = max(4, int(round((n / (a * a * b)) ** (1.0 / 3.0))))
    ny = max(4, int(round(nz * a)))
    return max(6, int(round(n / (ny * nz)))), ny, nz


# ------------------------------------------------------------------------------------------
# bodies
# ------------------------------------------------------------------------------------------
def _material(c):
    if c["mat"] == "BB":
        return pd.BBMaterial()
    if c["mat"] == "OSB":
        return pd.OSBMaterial(kernel=pd.cubic_b_spline_kernel if c.get("kernel") == "cubic"
                              else pd.linear_kernel)
    return pd.CMaterial(model=pd.NeoHooke() if c.get("model") == "neohooke" else
                        pd.SaintVenantKirchhoff(),
                        zem=pd.ZEMWan() if c.get("zem") == "wan" else pd.ZEMSilling())


def _tuned(c):
    return c["prec"] == "fp32" and (c["kind"] == "ensemble" or c["nx"] * c["ny"] * c["nz"] >= 100_000)


def _lattice(c, seed):
    """Positions (3, n), volumes and the lattice index of every point."""
    nx, ny, nz = c["nx"], c["ny"], c["nz"]
    pos, vol = pd.uniform_box(nx * DX, ny * DX, nz * DX, DX)
    if c.get("jitter"):
        g = torch.Generator().manual_seed(1000 + seed)
        j = torch.rand(pos.shape, generator=g, dtype=torch.float64).numpy()
        pos = pos + (2.0 * j - 1.0) * (c["jitter"] * DX)
    k = np.arange(nx * ny * nz)
    return pos, vol, (k % nx, (k // nx) % ny, k // (nx * ny))


def _velocity(c, seed, pos):
    """A smooth field of three standing waves with phases of the seed, 0.4 m/s in all."""
    r = np.random.default_rng(seed)
    size = np.array([c["nx"], c["ny"], c["nz"]])[:, None] * DX
    v = np.empty((pos.shape[1], 3))
    s = 2.0 * math.pi * (pos / size)
    for k in range(3):
        ph, w = r.uniform(0, 2 * math.pi, 3), r.uniform(0.05, 0.15, 3)
        v[:, k] = (w[0] * np.sin(s[0] + ph[0]) + w[1] * np.sin(s[1] + ph[1])
                   + w[2] * np.sin(s[2] + ph[2]))
    return v


def _speed(c, seed):
    """Speed of the pulled layers: 0.6 m/s, less for bodies that the layers would tear off from
    within the pass; 0.6 m/s for the plate, which is meant to break."""
    v = 0.6 if c.get("tear") else min(0.6, 0.3 * c["ny"] / c["steps"])
    return v * (1.0 + 0.2 * float(np.random.default_rng(seed + 77).random()))


def _crack(c, ix, iy):
    """Point masks of an edge crack along half the length of the body (bonds across it are
    left out): below and above mid-height."""
    a = (ix < c["nx"] // 2) & (iy < c["ny"] // 2)
    b = (ix < c["nx"] // 2) & (iy >= c["ny"] // 2)
    return a, b


def _kwargs(c, **kw):
    d = dict(horizon=c.get("m", 3.015) * DX, rho=RHO, E=YOUNG, Gc=GC)
    if c["mat"] != "BB":
        d["nu"] = NU
    d.update(kw)
    return d


def _pulled(c, seed):
    pos, vol, (ix, iy, iz) = _lattice(c, seed)
    body = pd.Body(_material(c), pos, vol)
    pd.material(body, **_kwargs(c))
    if c.get("crack"):
        a, b = _crack(c, ix, iy)
        pd.point_set(body, "crack_a", a)
        pd.point_set(body, "crack_b", b)
        pd.precrack(body, "crack_a", "crack_b", update_dmg=False)
    v = _speed(c, seed)
    pd.point_set(body, "bottom", iy == 0)
    pd.point_set(body, "top", iy == c["ny"] - 1)
    pd.velocity_bc(lambda t: -v, body, "bottom", "y")
    pd.velocity_bc(lambda t: v, body, "top", "y")
    return body


def _pinned(*shape):
    return torch.zeros(shape, dtype=torch.float64, pin_memory=True)


def _host(a):
    t = _pinned(*a.shape)
    t.copy_(torch.from_numpy(np.ascontiguousarray(a)))
    return t


# ------------------------------------------------------------------------------------------
# what a program has in hand
# ------------------------------------------------------------------------------------------
def prepare(case, seed):
    return {"vv": _prepare_vv, "relax": _prepare_relax, "newton": _prepare_newton,
            "ensemble": _prepare_ensemble, "static": _prepare_static}[case["kind"]](case, seed)


def _tune(c, dev):
    if _tuned(c):
        dev.set_mapping(1, 128)
        dev.set_pipeline(5)
    if c.get("graph"):
        dev.set_graph(c["graph"])


def _prepare_vv(c, seed):
    body = _pulled(c, seed)
    dev = pd.DeviceBody(body, precision=c["prec"])
    _tune(c, dev)
    dt = dev.stable_timestep(SAFETY)
    dev.force(0.0, dt)
    n = body.n_points
    return dict(case=c, dev=dev, dt=dt, x=_host(body._pos), u=_pinned(n, 3), a=_pinned(n, 3),
                v=_host(_velocity(c, seed, body.position)),
                out={"displacement": _pinned(n, 3), "velocity": _pinned(n, 3), "damage": _pinned(n)})


DR_STRAIN = 5e-5


def _relax_load(c, seed):
    """Force density on the x = max layer of the bar that strains it by about DR_STRAIN."""
    return DR_STRAIN * YOUNG / DX * (1.0 + 0.2 * float(np.random.default_rng(seed).random()))


def _prepare_relax(c, seed):
    pos, vol, (ix, iy, iz) = _lattice(c, seed)
    body = pd.Body(_material(c), pos, vol)
    pd.material(body, **_kwargs(c, Gc=1e4))
    b = _relax_load(c, seed)
    pd.point_set(body, "left", ix < 2)
    pd.point_set(body, "right", ix == c["nx"] - 1)
    for d in "xyz":
        pd.velocity_bc(lambda t: 0.0, body, "left", d)
    pd.forcedensity_bc(lambda t: b, body, "right", "x")
    n = body.n_points
    return dict(case=c, dev=pd.DeviceBody(body, precision=c["prec"]),
                solver=pd.DynamicRelaxation(steps=c["steps"]), x=_host(body._pos), u=_pinned(n, 3),
                out={"displacement": _pinned(n, 3), "velocity": _pinned(n, 3)})


def _beam_sets(c, pos):
    """The two supports (bottom lines near the ends) and the loaded line (top, mid-span)."""
    x, y = pos[0], pos[1]
    sup = np.minimum(np.abs(x - (x.min() + 5 * DX)), np.abs(x - (x.max() - 5 * DX))) < DX / 2
    top = np.abs(x) < 0.75 * DX
    return (np.abs(y - y.min()) < DX / 2) & sup, (np.abs(y - y.max()) < DX / 2) & top


def _beam_load(seed):
    return -2e-5 * (1.0 + 0.2 * float(np.random.default_rng(seed).random()))


def _prepare_newton(c, seed):
    pos, vol, _ = _lattice(c, seed)
    body = pd.Body(_material(c), pos, vol)
    kw = _kwargs(c)
    del kw["Gc"]
    pd.material(body, **kw)
    sup, top = _beam_sets(c, pos)
    pd.point_set(body, "support", sup)
    pd.point_set(body, "load", top)
    load = _beam_load(seed)
    for d in "xyz":
        pd.displacement_bc(lambda p: 0.0, body, "support", d)
    pd.displacement_bc(lambda p: load, body, "load", "y")
    dev = pd.DeviceBody(body, precision="fp64")
    # the reference's central rule for the products; every Newton correction solved to 1e-4
    nk = pd.NewtonKrylov(steps=1, tol=1e-9, tol_mode="relative", gmres_restart=50,
                         gmres_maxiter=8000, maxiter=20, preconditioner="block_poly")
    nkm.setup(dev, nk)
    n = body.n_points
    return dict(case=c, dev=dev, solver=nk, x=_host(body._pos), u=_pinned(n, 3),
                out={"displacement": _pinned(n, 3)})


def _specimens(c, seed):
    """(m, E, rho, crack length) of every specimen: 4m x 2m x m points."""
    r = np.random.default_rng(c["nx"] * 100 + c["specimens"])
    ms = [max(5, int(round(c["nx"] * f))) for f in r.uniform(0.7, 1.5, c["specimens"])]
    r = np.random.default_rng(seed)
    return [(m, r.uniform(50e9, 200e9), r.uniform(2000.0, 8000.0), r.uniform(0.1, 0.4)) for m in ms]


def _prepare_ensemble(c, seed):
    bodies = []
    v = _speed(dict(c, ny=2 * c["nx"]), seed)
    for m, E, rho, a in _specimens(c, seed):
        pos, vol, (ix, iy, iz) = _lattice(dict(nx=4 * m, ny=2 * m, nz=m), seed)
        body = pd.Body(_material(c), pos, vol)
        pd.material(body, **_kwargs(c, E=E, rho=rho))
        cut = ix < int(a * 4 * m)
        pd.point_set(body, "crack_a", cut & (iy < m))
        pd.point_set(body, "crack_b", cut & (iy >= m))
        pd.precrack(body, "crack_a", "crack_b", update_dmg=False)
        pd.point_set(body, "bottom", iy == 0)
        pd.point_set(body, "top", iy == 2 * m - 1)
        pd.velocity_bc(lambda t: -v, body, "bottom", "y")
        pd.velocity_bc(lambda t: v, body, "top", "y")
        bodies.append(body)
    ens = pd.Ensemble(bodies, precision=c["prec"], graph_steps=c["graph"], classes=c["classes"])
    ens.set_mapping(1, 128)
    for dev in ens.devs:
        dev.set_pipeline(5)
    zeros = [_pinned(dev.n, 3) for dev in ens.devs]
    return dict(case=c, ens=ens, zeros=zeros)


def _prepare_static(c, seed):
    pos, vol, _ = _lattice(c, seed)
    n = pos.shape[1]
    p = pd.point_parameters(_material(c), **_kwargs(c))
    x = np.ascontiguousarray(pos.T)
    delta = np.full(n, p.delta)
    lib = pd.lib()
    nb = ctypes.c_int64()
    args = (n, L.ptr(x), L.ptr(delta), None, 0, None, None)
    L.check(lib.pd_find_bonds(*args, 0, None, None, None, None, ctypes.byref(nb), 0))
    off, nbr = np.empty(n + 1, np.int64), np.empty(nb.value, np.int32)
    length, permit = np.empty(nb.value), np.empty(nb.value, np.uint8)
    L.check(lib.pd_find_bonds(*args, nb.value, L.ptr(off), L.ptr(nbr), L.ptr(length), L.ptr(permit),
                              ctypes.byref(nb), 0))
    v = _velocity(c, seed, pos)
    d = {k: torch.from_numpy(a).cuda() for k, a in dict(
        X=x, x=x + 2e-6 * v, vol=vol, off=off, nbr=nbr, length=length, permit=permit).items()}
    d["active"] = torch.ones(nb.value, dtype=torch.uint8, device="cuda")
    d["b_int"] = torch.empty((n, 3), dtype=torch.float64, device="cuda")
    d["n_active"] = torch.empty(n, dtype=torch.int64, device="cuda")
    return dict(case=c, n=n, params=p.to_c(), d=d)


# ------------------------------------------------------------------------------------------
# one pass
# ------------------------------------------------------------------------------------------
def run(state):
    return {"vv": _run_vv, "relax": _run_relax, "newton": _run_newton, "ensemble": _run_ensemble,
            "static": _run_static}[state["case"]["kind"]](state)


def _read(s, dev, names):
    """The fields read into the program's page-locked arrays; the FP32 form's as float32."""
    res = {}
    for k in names:
        t = s["out"][k]
        dev.field(k, out=t.numpy())
        res[k] = t.float() if s["case"]["prec"] == "fp32" else t
    return res


def _run_vv(s):
    c, dev = s["case"], s["dev"]
    u, v, a = s["u"].numpy(), s["v"].numpy(), s["a"].numpy()
    if c["prec"] == "fp64":
        dev.set_state(position=s["x"].numpy(), displacement=u, velocity=v, acceleration=a)
    else:
        dev.set_state(displacement=u, velocity=v, acceleration=a)
    dev.run(1, c["steps"], s["dt"])
    return _read(s, dev, ("displacement", "velocity", "damage"))


def _run_relax(s):
    dev, u = s["dev"], s["u"].numpy()
    dev.set_state(position=s["x"].numpy(), displacement=u, velocity=u, velocity_half=u)
    drm.solve(dev, s["solver"])
    return _read(s, dev, ("displacement", "velocity"))


def _run_newton(s):
    dev = s["dev"]
    dev.set_state(position=s["x"].numpy(), displacement=s["u"].numpy())
    s["solver"].stats.clear()
    nkm.step(dev, s["solver"], 1)
    return _read(s, dev, ("displacement",))


def _run_ensemble(s):
    c, ens = s["case"], s["ens"]
    for dev, z in zip(ens.devs, s["zeros"]):
        z = z.numpy()
        dev.set_state(displacement=z, velocity=z, acceleration=z)
    ens.run(c["steps"])
    res = {}
    for name in ("displacement", "velocity"):
        whole = [torch.from_numpy(np.ascontiguousarray(dev.field(name).T)).float() for dev in ens.devs]
        for k in range(len(ens.bodies)):
            g, q = ens.where[k]
            o = ens.offsets[g][q]
            res["%s%d" % (name, k)] = whole[g][o:o + ens.bodies[k].n_points]
    return res


def _run_static(s):
    d = s["d"]
    st = pd.lib().pd_osb_force_static(
        s["n"], d["X"].data_ptr(), d["x"].data_ptr(), d["vol"].data_ptr(), d["off"].data_ptr(),
        d["nbr"].data_ptr(), d["length"].data_ptr(), d["permit"].data_ptr(), d["active"].data_ptr(),
        ctypes.byref(s["params"]), L.KERNEL_LINEAR, d["b_int"].data_ptr(), d["n_active"].data_ptr(),
        torch.cuda.current_stream().cuda_stream)
    L.check(st)
    return {"b_int": d["b_int"], "n_active": d["n_active"], "active": d["active"]}


# ------------------------------------------------------------------------------------------
# the work of a pass
# ------------------------------------------------------------------------------------------
def _offsets(m, jitter=0.0):
    """Lattice offsets of the points that may lie within m (and the jitter) of a point."""
    r = m + 2.0 * math.sqrt(3.0) * jitter
    k = int(math.floor(r))
    return [(a, b, g) for g in range(-k, k + 1) for b in range(-k, k + 1) for a in range(-k, k + 1)
            if 0 < a * a + b * b + g * g <= r * r + 1e-9]


def _bonds(nx, ny, nz, m):
    return sum(max(0, nx - abs(a)) * max(0, ny - abs(b)) * max(0, nz - abs(g))
               for a, b, g in _offsets(m))


# per directed bond and evaluation: neighbour index and state bit (the bond vector and length
# follow from the points); operations of the failure test and the force
BOND_BYTES = 4.0 + 0.125
BOND_FLOPS = {"BB": 25.0, "OSB": 55.0, "C": 130.0}
# per point and step: displacement, velocity and force state read and written
POINT_BYTES = {"fp32": 140.0, "fp64": 184.0}
POINT_EXTRA = {"BB": 0.0, "OSB": 8.0, "C": 72.0}


def work(case):
    c = case
    m = c.get("m", 3.015)
    if c["kind"] == "ensemble":
        boxes = [(4 * k, 2 * k, k) for k, _, _, _ in _specimens(c, 0)]
    else:
        boxes = [(c["nx"], c["ny"], c["nz"])]
    nb = sum(_bonds(*b, m) for b in boxes)
    n = sum(a * b * g for a, b, g in boxes)
    steps = {"static": 1, "newton": 400}.get(c["kind"]) or c["steps"]
    per = nb * BOND_BYTES + n * (POINT_BYTES[c["prec"]] + POINT_EXTRA[c["mat"]])
    return {"bytes": steps * per, "flops": steps * nb * BOND_FLOPS[c["mat"]]}


# ------------------------------------------------------------------------------------------
# the same results in plain torch, FP64
# ------------------------------------------------------------------------------------------
EXACT_POINTS = 1_100_000


class _Plain:
    """Bonds as an (n, k) table of neighbours from the lattice offsets, force densities by
    dense sums over it, in chunks of points."""

    def __init__(self, c, seed, kw=None, crack=None):
        self.c = c
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        pos, vol, (ix, iy, iz) = _lattice(c, seed)
        self.p = pd.point_parameters(_material(c), **(kw or _kwargs(c)))
        self.ix, self.iy, self.iz = ix, iy, iz
        t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(self.dev)  # noqa: E731
        self.X, self.V = t(pos.T), t(vol)
        n = self.n = pos.shape[1]
        nx, ny, nz = c["nx"], c["ny"], c["nz"]
        offs = _offsets(c.get("m", 3.015), c.get("jitter", 0.0))
        I = [t(a) for a in (ix, iy, iz)]
        J, M, LN = [], [], []
        own = torch.arange(n, device=self.dev)
        masks = None if crack is None else [t(a) for a in crack]
        for a, b, g in offs:
            ok = ((I[0] + a >= 0) & (I[0] + a < nx) & (I[1] + b >= 0) & (I[1] + b < ny)
                  & (I[2] + g >= 0) & (I[2] + g < nz))
            j = torch.where(ok, own + (a + nx * (b + ny * g)), own)
            d = self.X[j] - self.X
            l2 = (d * d).sum(1)
            ok &= l2 <= self.p.delta ** 2
            if masks is not None:
                A, B = masks
                ok &= ~((A & B[j]) | (B & A[j]))
            J.append(torch.where(ok, j, own).int())
            M.append(ok)
            LN.append(torch.where(ok, l2.sqrt(), torch.ones_like(l2)))
        self.J, self.active = torch.stack(J, 1), torch.stack(M, 1)
        self.L = torch.stack(LN, 1)
        self.count = self.active.sum(1)
        self.fails = self.p.has_fracture
        self.chunk = max(1, 8_000_000 // len(offs))
        self.u = torch.zeros_like(self.X)

    def chunks(self):
        for a in range(0, self.n, self.chunk):
            yield slice(a, min(self.n, a + self.chunk))

    def geometry(self, s):
        """Neighbours, bond vectors, displacement differences, reference and current lengths
        and the extension l - L without its cancellation."""
        j = self.J[s].long()
        xi = self.X[j] - self.X[s, None]
        du = self.u[j] - self.u[s, None]
        Ln = self.L[s]
        l = (xi + du).square().sum(2).sqrt()
        return j, xi, du, l, Ln, ((2.0 * xi + du) * du).sum(2) / (l + Ln)

    def fail(self, s, e, Ln):
        if self.fails:
            self.active[s] &= ~(e / Ln > self.p.epsilon_c)
        return self.active[s].double()

    def omega(self, Ln):
        if self.c["mat"] == "OSB" and self.c.get("kernel") == "cubic":
            q = Ln / self.p.delta
            near = 2.0 / 3.0 - 4.0 * q ** 2 + 4.0 * q ** 3
            far = 4.0 / 3.0 - 4.0 * q + 4.0 * q ** 2 - 4.0 / 3.0 * q ** 3
            return torch.where(q <= 0.5, near, far)
        return self.p.delta / Ln

    def force(self):
        return {"BB": self._bb, "OSB": self._osb, "C": self._cmat}[self.c["mat"]]()

    def _bb(self):
        b = torch.empty_like(self.X)
        for s in self.chunks():
            j, xi, du, l, Ln, e = self.geometry(s)
            w = self.fail(s, e, Ln) * self.p.bc * e / Ln * self.V[j] / l.clamp_min(1e-300)
            b[s] = (w[..., None] * (xi + du)).sum(1)
        return b

    def _osb(self):
        p = self.p
        c1, c2 = torch.zeros(2, self.n, dtype=torch.float64, device=self.dev)
        for s in self.chunks():
            j, xi, du, l, Ln, e = self.geometry(s)
            w = self.fail(s, e, Ln) * self.omega(Ln) * self.V[j]
            m = (w * Ln * Ln).sum(1)
            some = m != 0.0
            m = torch.where(some, m, torch.ones_like(m))
            th = 3.0 / m * (w * Ln * e).sum(1)
            c1[s] = torch.where(some, 15.0 * p.G / m, 0.0)
            c2[s] = torch.where(some, th * (3.0 * p.K / m - c1[s] / 3.0), 0.0)
        b = torch.empty_like(self.X)
        for s in self.chunks():
            j, xi, du, l, Ln, e = self.geometry(s)
            f = (c2[s, None] + c2[j]) * Ln + (c1[s, None] + c1[j]) * e
            f = self.active[s].double() * self.omega(Ln) * f * self.V[j] / l.clamp_min(1e-300)
            b[s] = (f[..., None] * (xi + du)).sum(1)
        return b

    def _cmat(self):
        """With H = F - I and the stabilising stiffness S, the bond force of a point is
        w (P K^-1 xi + S (eta - F xi)) = w (A xi + S du), A = P K^-1 - S H."""
        p = self.p
        A = torch.empty((self.n, 3, 3), dtype=torch.float64, device=self.dev)
        S = torch.empty_like(A)
        eye = torch.eye(3, dtype=torch.float64, device=self.dev)
        for s in self.chunks():
            j, xi, du, l, Ln, e = self.geometry(s)
            w = (self.fail(s, e, Ln) * self.omega(Ln) * self.V[j])[..., None]
            Ki = torch.linalg.inv((w * xi).transpose(1, 2) @ xi)
            H = ((w * du).transpose(1, 2) @ xi) @ Ki
            F = eye + H
            E = 0.5 * (H + H.transpose(1, 2) + H.transpose(1, 2) @ H)
            if self.c.get("model") == "neohooke":
                Ci = torch.linalg.inv(eye + 2.0 * E)
                lj = p.lambda_ * torch.log(torch.linalg.det(F))
                T = Ci @ (2.0 * p.mu * E + lj[:, None, None] * eye)
            else:
                tr = E.diagonal(dim1=1, dim2=2).sum(1)
                T = p.lambda_ * tr[:, None, None] * eye + 2.0 * p.mu * E
            if self.c.get("zem") == "wan":
                tr = Ki.diagonal(dim1=1, dim2=2).sum(1)
                S[s] = p.lambda_ * tr[:, None, None] * eye + p.mu * (Ki + Ki.transpose(1, 2))
            else:
                S[s] = 0.5 * p.bc / p.delta * eye
            A[s] = F @ T @ Ki - S[s] @ H
        b = torch.empty_like(self.X)
        for s in self.chunks():
            j, xi, du, l, Ln, e = self.geometry(s)
            w = self.active[s].double() * self.omega(Ln) * self.V[j]
            t = ((A[s, None] + A[j]) * xi[:, :, None]).sum(3)
            if self.c.get("zem") == "wan":
                t += ((S[s, None] + S[j]) * du[:, :, None]).sum(3)
            else:
                t += p.bc / p.delta * du
            b[s] = (w[..., None] * t).sum(1)
        return b

    def stable_step(self):
        s = (self.active.double() * self.V[self.J.long()] * self.p.bc / self.L).sum(1)
        return SAFETY * float(torch.sqrt(2.0 * self.p.rho / s).min())

    def verlet(self, v, ends, speed, steps, dt):
        a = torch.zeros_like(v)
        for _ in range(steps):
            vh = v + a * (0.5 * dt)
            vh[ends[0], 1] = -speed
            vh[ends[1], 1] = speed
            self.u += vh * dt
            a = self.force() / self.p.rho
            v = vh + a * (0.5 * dt)
        damage = 1.0 - self.active.sum(1).double() / self.count.double()
        return {"displacement": self.u, "velocity": v, "damage": damage}

    def ends(self):
        return [torch.from_numpy(np.nonzero(self.iy == k)[0]).to(self.dev)
                for k in (0, self.c["ny"] - 1)]


def exact(case, seed):
    c = case
    if c["kind"] == "ensemble":
        return _exact_ensemble(c, seed)
    # the cubes of steps and bonds that the dense sums get through in the time there is
    n = c["nx"] * c["ny"] * c["nz"]
    if n * c.get("steps", 1) > 45 * EXACT_POINTS or n > EXACT_POINTS:
        return None
    return {"vv": _exact_vv, "relax": _exact_relax, "newton": _exact_newton,
            "static": _exact_static}[c["kind"]](c, seed)


def _exact_vv(c, seed):
    if c["nx"] * c["ny"] * c["nz"] * c["steps"] > {"BB": 45e6, "OSB": 45e6, "C": 12e6}[c["mat"]]:
        return None
    pos, _, (ix, iy, _) = _lattice(c, seed)
    P = _Plain(c, seed, crack=_crack(c, ix, iy) if c.get("crack") else None)
    v = torch.from_numpy(_velocity(c, seed, pos)).to(P.dev)
    return P.verlet(v, P.ends(), _speed(c, seed), c["steps"], P.stable_step())


def _exact_ensemble(c, seed):
    res = {}
    v = _speed(dict(c, ny=2 * c["nx"]), seed)
    for k, (m, E, rho, a) in enumerate(_specimens(c, seed)):
        b = dict(c, nx=4 * m, ny=2 * m, nz=m)
        P = _Plain(b, seed, kw=_kwargs(c, E=E, rho=rho), crack=_ensemble_crack(b, a, m))
        out = P.verlet(torch.zeros_like(P.X), P.ends(), v, c["steps"], P.stable_step())
        for name in ("displacement", "velocity"):
            res["%s%d" % (name, k)] = out[name]
    return res


def _ensemble_crack(b, a, m):
    _, _, (ix, iy, _) = _lattice(dict(b, jitter=0.0), 0)
    cut = ix < int(a * 4 * m)
    return cut & (iy < m), cut & (iy >= m)


def _exact_relax(c, seed):
    P = _Plain(c, seed, kw=_kwargs(c, Gc=1e4))
    left = torch.from_numpy(P.ix < 2).to(P.dev)
    bext = torch.zeros_like(P.X)
    bext[torch.from_numpy(P.ix == c["nx"] - 1).to(P.dev), 0] = _relax_load(c, seed)
    lam = (0.25 * P.count.double() * (5.0 * math.pi * P.p.delta ** 2 * P.p.bc))[:, None]
    vh, vho, bo = (torch.zeros_like(P.X) for _ in range(3))
    v = torch.zeros_like(P.X)
    for step in range(1, c["steps"] + 1):
        vh[left] = 0.0
        P.u += vh
        b = P.force()
        if step == 1:
            vh = 0.5 * (b + bext) / lam
        else:
            free = vh != 0.0
            num = float((-(P.u[free] ** 2) * (b - bo)[free] / (lam.expand_as(vho) * vho)[free]).sum())
            den = float((P.u ** 2).sum())
            cn = 2.0 * math.sqrt(num / den) if den != 0.0 and num / den > 0.0 else 0.0
            cn = 1.9 if cn > 2.0 else cn
            vh = ((2.0 - cn) * vho + 2.0 * (b + bext) / lam) / (2.0 + cn)
        v = 0.5 * (vho + vh)
        vho, bo = vh.clone(), b
    return {"displacement": P.u, "velocity": v}


def _exact_newton(c, seed):
    """Newton's method with the exact tangent; the linear systems by conjugate gradients."""
    kw = _kwargs(c)
    del kw["Gc"]
    P = _Plain(c, seed, kw=kw)
    pos = P.X.t().cpu().numpy()
    sup, top = (torch.from_numpy(a).to(P.dev) for a in _beam_sets(c, pos))
    free = torch.ones_like(P.X)
    free[sup] = 0.0
    free[top, 1] = 0.0
    P.u[top, 1] = _beam_load(seed)
    s = slice(0, P.n)
    for _ in range(30):
        j, xi, du, l, Ln, e = P.geometry(s)
        eta = xi + du
        l = torch.where(P.active, l, torch.ones_like(l))
        act = P.active.double() * P.p.bc * P.V[j] * P.V[:, None]
        f = act * e / (Ln * l)
        r = free * (f[..., None] * eta).sum(1)
        size = float(r.norm())
        first = size if _ == 0 else first
        if size <= 2e-14 * first:
            break
        q = act / l ** 3

        def stiff(d):
            dd = d[j] - d[:, None]
            t = f[..., None] * dd + (q * (eta * dd).sum(2))[..., None] * eta
            return -free * t.sum(1)

        diag = ((f[..., None] + q[..., None] * eta * eta).sum(1)).clamp_min(1e-300)
        d, res = torch.zeros_like(r), r.clone()
        z = free * res / diag
        w, rz = z.clone(), float((res * z).sum())
        for _k in range(4000):
            Aw = stiff(w)
            al = rz / float((w * Aw).sum())
            d += al * w
            res -= al * Aw
            if float(res.norm()) <= 1e-10 * size:
                break
            z = free * res / diag
            rz, be = float((res * z).sum()), rz
            w = z + (rz / be) * w
        P.u += d
    return {"displacement": P.u}


def _exact_static(c, seed):
    P = _Plain(c, seed)
    pos = P.X.t().cpu().numpy()
    P.u = 2e-6 * torch.from_numpy(_velocity(c, seed, pos)).to(P.dev)
    b = P.force()
    return {"b_int": b, "n_active": None, "active": None}
