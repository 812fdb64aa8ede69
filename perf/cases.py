"""The work that programs built on this library have it do, as timed cases.

Every case goes through the public entry points (the Python binding's classes,
or the C ABI's device-pointer functions for the column and flux kernels), as
the tests, the bench and the reference's drivers do:

* ``step``     a forecast member advanced a few steps from its analysis
               (device snapshot, RK3 with vertically implicit substeps)
* ``nested``   one parent step of a two-way nested set
* ``helmholtz``the semi-implicit step's elliptic solve over a hill
* ``window``   the tangent-linear or the adjoint of an assimilation window
* ``columns``  batched tridiagonal column solves
* ``flux``     flux-form scalar advection
* ``monitor``  the time-step control and budget reductions of a driver loop

Mixed-precision models compute in single precision; their results are taken
in single precision, the type a history file stores. FP64 results are the
device's own doubles.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "vibe-model_gb300"))
import vibe_gb300 as vg  # noqa: E402

G, RD, CP, CV, EPS, P00 = 9.80665, 287.05, 1004.64, 717.63, 0.62197, 100000.0
F64 = torch.float64
U, V, W, RHO, TH, PI, QV = range(7)
# first-layer to top stretching ratios of the bench's 80, 60 and 50 level grids
STRETCH = {80: 1.0341247533415947, 60: 1.0530384502435775}


def listed():
    return [
        # the smallest forecast: the 64 x 64 x 40 warm-bubble grid, launch-bound
        dict(name="step_bubble", kind="step", nx=64, ny=64, nz=40, dx=250.0, z_top=10000.0, dt=2.0, steps=4,
             mixed=True, moist=False),
        # a nest-sized member of ragged extent
        dict(name="step_ragged", kind="step", nx=193, ny=193, nz=60, dx=1000.0, z_top=20000.0, dt=6.0, steps=4,
             mixed=True, moist=False),
        # the headline single domain
        dict(name="step_domain", kind="step", nx=512, ny=512, nz=80, dx=1000.0, z_top=20000.0, dt=6.0, steps=4,
             mixed=True, moist=False),
        # the plain FP64 path, used where results have to track the reference
        dict(name="step_fp64", kind="step", nx=128, ny=128, nz=80, dx=1000.0, z_top=20000.0, dt=6.0, steps=1,
             mixed=False, moist=False),
        # moisture prognostic, Kessler warm rain at every stage
        dict(name="step_moist", kind="step", nx=256, ny=256, nz=80, dx=1000.0, z_top=20000.0, dt=6.0, steps=2,
             mixed=True, moist=True),
        # a parent with two ragged r = 3 nests, one parent step (one graph)
        dict(name="nested", kind="nested", nx=192, ny=192, nz=60, cnx=193, cny=130, dnx=97, dny=241),
        # the semi-implicit solve over the hill, to 1e-10
        dict(name="helmholtz", kind="helmholtz", nx=256, ny=256, nz=64),
        # an outer loop's tangent-linear sweep. Windows are FP64, the models'
        # default: a single-precision trajectory rounds |w| across the upwind
        # switch at 1e-3 m/s, where the derivative jumps, so that two roundings
        # of it differ by more than the arithmetic does
        dict(name="window_tl", kind="window", nx=96, ny=96, nz=50, steps=3, every=2, mixed=False, adjoint=False),
        # the gradient sweep, with recomputation from checkpoints
        dict(name="window_ad", kind="window", nx=64, ny=72, nz=50, steps=3, every=2, mixed=False, adjoint=True),
        # every column of the headline domain solved once
        dict(name="columns", kind="columns", n=80, systems=262144, f64=True),
        # scalar advection of a nest-to-domain sized field over terrain
        dict(name="flux", kind="flux", nx=384, ny=384, nz=60, f64=True, terrain=True),
        # CFL scan and compensated mass sum, once per driver step
        dict(name="monitor", kind="monitor", nx=384, ny=384, nz=60, f64=True, terrain=True),
    ]


def draw(rng):
    def logi(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["step", "step", "step", "nested", "helmholtz", "window", "window", "columns", "columns",
                       "flux", "monitor"])
    if kind == "step":
        mixed = rng.random() < 0.75
        moist = mixed and rng.random() < 0.25
        hi = 288 if moist else 400 if mixed else 120
        return dict(kind=kind, nx=logi(40, hi), ny=logi(40, hi), nz=rng.randint(30, 80), dx=1000.0, z_top=20000.0,
                    dt=6.0, steps=rng.randint(1, 4) if mixed else 1, mixed=mixed, moist=moist)
    if kind == "nested":
        return dict(kind=kind, nx=rng.randint(140, 256), ny=rng.randint(140, 256), nz=rng.randint(30, 60),
                    cnx=rng.randint(60, 200), cny=rng.randint(60, 150), dnx=rng.randint(60, 200),
                    dny=rng.randint(60, 150))
    if kind == "helmholtz":
        return dict(kind=kind, nx=logi(48, 256), ny=logi(48, 256), nz=rng.randint(24, 64))
    if kind == "window":
        return dict(kind=kind, nx=logi(32, 96), ny=logi(32, 80), nz=rng.randint(24, 50), steps=rng.randint(1, 3),
                    every=2, mixed=False, adjoint=rng.random() < 0.5)
    if kind == "columns":
        n = logi(6, 320)
        return dict(kind=kind, n=n, systems=min(262144, logi(600, 20_000_000 // n)), f64=rng.random() < 0.6)
    return dict(kind=kind, nx=logi(48, 512), ny=logi(48, 512), nz=rng.randint(20, 80), f64=rng.random() < 0.7,
                terrain=rng.random() < 0.7)


# ---- grids, base state and perturbed states (the library's set-up formulas) ----
def stretch_of(nz):
    return STRETCH.get(nz, 1.03)


def zeta_of(nz):
    dz = stretch_of(nz) ** np.arange(nz)
    z = np.concatenate([[0.0], np.cumsum(dz) / dz.sum()])
    z[-1] = 1.0
    return z


def base_of(zeta, z_top, bv_n=0.01):
    """theta0, pi0, rho0 per level of the N = 0.01 profile, 250 m table."""
    zp = np.arange(int(math.ceil(z_top / 250.0)) + 2) * 250.0
    tab = 300.0 * np.exp(bv_n * bv_n * zp / G)
    zi = zeta * z_top
    th = np.interp(zi, zp, tab)
    thm = 0.5 * (th[:-1] + th[1:])
    pi = 1.0 - np.cumsum(G * np.diff(zi) / (CP * thm))
    return thm, pi, P00 * pi ** (CV / RD) / (RD * thm)


def gen_of(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def member(nx, ny, nz, dx, z_top, seed, moist=False, waves=False):
    """A perturbed member: theta' noise below 1 km and 20 warm bubbles, wind
    noise on u = 10 m/s, pi from the equation of state. waves: instead of the
    noise, resolved waves of theta' and w at every height and a wind across
    the grid (the state an assimilation cycle linearises about)."""
    g = gen_of(seed)

    def rand(*s):
        return torch.rand(*s, dtype=F64, device="cuda", generator=g)

    def randn(*s):
        return torch.randn(*s, dtype=F64, device="cuda", generator=g)

    zeta = zeta_of(nz)
    th0, pi0, rho0 = (torch.tensor(a, dtype=F64, device="cuda")[:, None, None] for a in base_of(zeta, z_top))
    zc = torch.tensor(0.5 * (zeta[:-1] + zeta[1:]) * z_top, dtype=F64, device="cuda")
    th = th0.expand(nz, ny, nx).clone()
    if not waves:
        low = zc < 1000.0
        th[low] += rand(int(low.sum()), ny, nx) - 0.5
    x = (torch.arange(nx, dtype=F64, device="cuda") + 0.5) * dx
    y = (torch.arange(ny, dtype=F64, device="cuda") + 0.5) * dx
    par = torch.rand(20, 5, dtype=F64, generator=torch.Generator().manual_seed(seed))
    for a, r, cx, cy, cz in par.tolist():
        r = 1000.0 + 3000.0 * r
        r2 = (((x - cx * nx * dx) / r) ** 2)[None, None, :] + (((y - cy * ny * dx) / r) ** 2)[None, :, None] + \
            (((zc - 1000.0 - 4000.0 * cz) / r) ** 2)[:, None, None]
        th += (1.0 + 2.0 * a) * torch.cos(0.5 * math.pi * r2.clamp(max=1.0).sqrt()) ** 2
    u = 10.0 + 0.5 * randn(nz, ny, nx + 1)
    v = (4.0 if waves else 0.0) + 0.5 * randn(nz, ny + 1, nx)
    w = torch.zeros(nz + 1, ny, nx, dtype=F64, device="cuda")
    w[1:-1] = 0.05 * randn(nz - 1, ny, nx)
    if waves:
        kk = torch.arange(nz + 1, dtype=F64, device="cuda")[:, None, None]
        jj = torch.arange(ny, dtype=F64, device="cuda")[:, None]
        ii = torch.arange(nx, dtype=F64, device="cuda")
        u, v = 10.0 + 0.2 * (u - 10.0), 4.0 + 0.2 * (v - 4.0)
        w *= 0.02
        par = torch.rand(5, 7, dtype=F64, generator=torch.Generator().manual_seed(seed + 1))
        for a, b, c, sx, sy, ph, amp in par.tolist():
            wave = torch.sin(2 * math.pi * (ii * (1 if sx < 0.5 else -1) / (8 + 12 * a) +
                                            jj * (1 if sy < 0.5 else -1) / (8 + 12 * b) + kk / (8 + 12 * c) + ph))
            th += (0.3 + 0.7 * amp) * wave[:nz]
            w[1:-1] += 0.05 * amp * wave[1:-1]
        th += 0.01 * randn(nz, ny, nx)
    rho = rho0.expand(nz, ny, nx).clone()
    if moist:
        qv = (0.025 * torch.exp(-zc / 2500.0))[:, None, None].expand(nz, ny, nx).clone()
    else:
        qv = torch.zeros(nz, ny, nx, dtype=F64, device="cuda")
    pi = (rho * RD * th * ((1.0 + qv / EPS) / (1.0 + qv)) / P00) ** (RD / CV)
    return [u, v, w, rho, th, pi, qv]


def setup_of(nx, ny, nz, dx, z_top, moist=False, beta=0.5, rigid=0):
    return vg.Setup.defaults(nx=nx, ny=ny, nz=nz, dx=dx, dy=dx, z_top=z_top, zeta_first=50.0,
                             zeta_stretch=stretch_of(nz), ref_kind=1, theta0=300.0, bv_n=0.01, profile_dz=250.0,
                             bubble_amplitude=0.0, qv_surface=0.0, u_background=10.0, shear_u=0.0, advection=5,
                             weno_scalars=1, weno_advective=1, pgf_perturbation=1, split_fast=1, acoustic_mode=2,
                             hevi_beta=beta, w_rigid=rigid, moist=1 if moist else 0, coriolis=0)


def storage(setup, fields):
    """The fields as host arrays in the library's halo'd storage layout."""
    out = []
    for sp, f in enumerate(fields):
        a = torch.zeros(vg.storage_shape(setup, sp), dtype=F64, pin_memory=True)
        a[4:-4, 4:-4, 4:-4].copy_(f)
        out.append(a)
    return out


def model_of(setup, mixed, fields):
    m = vg.Model(setup, vg.MIXED if mixed else vg.FP64)
    arrays = storage(setup, fields)
    m.set_state_ptrs([a.data_ptr() for a in arrays])
    m.sync()
    return m


class _Mem:
    """A model's device buffer; keeps the model while a tensor over it lives."""

    def __init__(self, model, ptr, shape):
        self.model = model
        self.__cuda_array_interface__ = dict(shape=shape, typestr="<f8", data=(ptr, False), version=3, strides=None)


class Nested(vg.Nested):
    def __del__(self):
        self.close()


class Window(vg.Window):
    def __del__(self):
        self.close()


def fields_of(m, species, single):
    """The model's current fields on the device (interior boxes)."""
    s, out = m.setup, []
    for sp in species:
        ptr, pitch = ctypes.POINTER(ctypes.c_double)(), ctypes.c_int()
        if vg.lib.vibe_gb300_device_field(m.h, sp, ctypes.byref(ptr), ctypes.byref(pitch)):
            raise RuntimeError(vg.lib.vibe_gb300_last_error().decode())
        t = torch.as_tensor(_Mem(m, ctypes.cast(ptr, ctypes.c_void_p).value, (s.nz + 1, s.ny + 1, pitch.value)),
                            device="cuda")
        t = t[:s.nz + (sp == W), :s.ny + (sp == V), :s.nx + (sp == U)]
        out.append(t.to(torch.float32) if single else t)
    return out


# ---- the C ABI's device-pointer functions ----
_P, _I, _Z = ctypes.c_void_p, ctypes.c_int, ctypes.c_size_t
_c = {}
for _t, _real in (("f64", ctypes.c_double), ("f32", ctypes.c_float)):
    for _name, _args in (("tridiagonal_solve_batched", [_P] * 4 + [_I, _I, _P, _P, _P]),
                         ("cfl_scan", [_P] * 5 + [_I] * 3 + [_real] * 4 + [_P, _P]),
                         ("neumaier_sum", [_P, _Z, _P, _P]),
                         ("advect_scalar_flux", [_P] * 7 + [_I] * 3 + [_real] * 3 + [_P, _P])):
        _f = getattr(ctypes.CDLL(vg.LIB_PATH), "vibe_%s_%s_dev" % (_name, _t))
        _f.restype, _f.argtypes = _I, _args
        _c[_name, _t] = _f


def _ok(rc):
    if rc:
        raise RuntimeError("rc=%d: %s" % (rc, vg.lib.vibe_c_last_error().decode()))


def cells_of(c):
    return c["nx"] * c["ny"] * c["nz"]


# ---- inputs ----
def column_inputs(c, seed):
    g, n, s = gen_of(seed), c["n"], c["systems"]
    dt = F64 if c["f64"] else torch.float32

    def rand(*shape):
        return torch.rand(*shape, dtype=dt, device="cuda", generator=g)

    # the implicit vertical operator: diagonally dominant, of varying strength
    a, k = -3.0 * rand(s, n - 1), -3.0 * rand(s, n - 1)
    b = 1.0 + 0.5 * rand(s, n)
    b[:, 1:] -= a
    b[:, :-1] -= k
    return a, b, k, rand(s, n) - 0.5


def grid_inputs(c, seed):
    g = gen_of(seed)
    dt = F64 if c["f64"] else torch.float32
    sh = (c["nz"], c["ny"], c["nx"])

    def rand(*shape):
        return torch.rand(*shape, dtype=dt, device="cuda", generator=g)

    u, v, w = 40.0 * rand(*sh) - 15.0, 30.0 * rand(*sh) - 15.0, 4.0 * rand(*sh) - 2.0
    q, rho = 300.0 + 5.0 * rand(*sh), 0.2 + rand(*sh)
    dzeta = torch.tensor(np.diff(zeta_of(c["nz"])), dtype=dt, device="cuda")
    zs = 800.0 * rand(c["ny"], c["nx"]) if c["terrain"] else None
    return dict(u=u, v=v, w=w, q=q, rho=rho, dzeta=dzeta, zs=zs)


def hill_inputs(c, seed):
    """The semi-implicit operator and right-hand side over a Gaussian hill."""
    nx, ny, nz = c["nx"], c["ny"], c["nz"]
    z = np.linspace(0.0, 1.0, nz + 1)
    x = (np.arange(nx) + 0.5) * 2000.0 - nx * 1000.0
    y = (np.arange(ny) + 0.5) * 2000.0 - ny * 1000.0
    zs = 800.0 * np.exp(-(x[None, :] ** 2 + y[:, None] ** 2) / 1e8)
    g = gen_of(seed)
    th0, pi0, _ = (torch.tensor(a, dtype=F64, device="cuda")[:, None, None] for a in base_of(z, 20000.0))
    th = th0 + torch.randn(nz, ny, nx, dtype=F64, device="cuda", generator=g) * 0.3
    a = 225.0 * (RD / CV) * pi0 * CP * th
    f = pi0 + 1e-3 * torch.randn(nz, ny, nx, dtype=F64, device="cuda", generator=g)
    return np.diff(z), zs, a.contiguous(), torch.ones_like(a), f.contiguous()


WIN = dict(dx=3000.0, z_top=20000.0, dt=15.0, beta=0.6, rigid=1)


def window_inputs(c, seed):
    nx, ny, nz = c["nx"], c["ny"], c["nz"]
    state = member(nx, ny, nz, WIN["dx"], WIN["z_top"], seed, waves=True)
    g = gen_of(seed + 77)
    amp = [1.0, 1.0, 0.1, 1e-4, 0.5, 1.4e-4, 0.0]
    pert = [s * torch.randn(f.shape, dtype=F64, device="cuda", generator=g) for s, f in zip(amp, state)]
    return state, pert


def nest_boxes(c):
    """Two nests beside each other in the parent: (nx, ny, i0, j0 in parent points)."""
    a, b = (c["cnx"], c["cny"]), (c["dnx"], c["dny"])
    return [(a[0], a[1], 20, 20), (b[0], b[1], 24, 28 + a[1] // 3)]


def prepare(case, seed):
    k = case["kind"]
    if k == "step":
        s = setup_of(case["nx"], case["ny"], case["nz"], case["dx"], case["z_top"], case["moist"])
        m = model_of(s, case["mixed"], member(s.nx, s.ny, s.nz, s.dx, s.z_top, seed, case["moist"]))
        if case["moist"]:
            m.set_physics_kessler(vg.Kessler.defaults(exner_offset=0))
        m.save_snapshot()
        return dict(case=case, m=m, stream=torch.cuda.ExternalStream(m.stream()))
    if k == "nested":
        base = dict(nz=case["nz"], z_top=20000.0)
        ps = setup_of(case["nx"], case["ny"], dx=3000.0, **base)
        fields = member(ps.nx, ps.ny, ps.nz, ps.dx, ps.z_top, seed)
        parent = model_of(ps, True, fields)
        host = [a.numpy() for a in storage(ps, fields)]
        children, ip, rp = [], [], []
        for nx, ny, i0, j0 in nest_boxes(case):
            cs = setup_of(nx, ny, dx=1000.0, **base)
            a, b = vg.NestPlacement(), vg.NestPlacement()
            a.i0, a.j0, a.ratio, a.boundary_zone, a.two_way = 3 * i0, 3 * j0, 3, 5, 1
            b.i0, b.j0, b.iext, b.jext, b.ratio, b.boundary_zone, b.two_way = i0, j0, nx // 3, ny // 3, 3, 5, 1
            ch = vg.Model(cs, vg.MIXED)
            st = [np.zeros(vg.storage_shape(cs, q)) for q in range(7)]
            vg.nest_interpolate_from_parent(a, [1, 2, 3, 0, 0, 0, 0], (ps.nx, ps.ny, ps.nz), host,
                                            (cs.nx, cs.ny, cs.nz), st)
            ch.set_state_ptrs([t.ctypes.data for t in st])
            ch.sync()
            children.append(ch)
            ip.append(a)
            rp.append(b)
        n = Nested([parent], children, [0, 0], ip, rp)
        models = [parent] + children
        for m in models:
            m.save_snapshot()
            m.sync()
        return dict(case=case, n=n, models=models, stream=torch.cuda.ExternalStream(n.stream()))
    if k == "helmholtz":
        dz, zs, a, b, f = hill_inputs(case, seed)
        h = vg.Helmholtz(vg.HZ_MG_BICGSTAB_MIXED, case["nx"], case["ny"], case["nz"], 2000.0, 2000.0, 20000.0, dz, zs,
                         200, 1e-10)
        st = torch.cuda.current_stream().cuda_stream
        torch.cuda.synchronize()
        h.set_coefficients_dev(a.data_ptr(), b.data_ptr(), st)
        return dict(case=case, h=h, keep=(a, b), f=f, x=torch.empty_like(f))
    if k == "window":
        s = setup_of(case["nx"], case["ny"], case["nz"], WIN["dx"], WIN["z_top"], beta=WIN["beta"],
                     rigid=WIN["rigid"])
        state, pert = window_inputs(case, seed)
        m = model_of(s, case["mixed"], state)
        w = Window(m, None, WIN["dt"], 6, case["steps"], case["every"])
        host = [a.numpy().ravel().copy() for a in storage(s, pert)]
        host += [np.zeros(host[QV].size) for _ in range(5)]
        return dict(case=case, m=m, w=w, pert=host)
    if k == "columns":
        a, b, c, d = column_inputs(case, seed)
        return dict(case=case, a=a, b=b, c=c, d=d, x=torch.empty_like(b))
    s = grid_inputs(case, seed)
    s["case"] = case
    if k == "flux":
        s["out"] = torch.empty_like(s["q"])
    else:
        s["cfl"], s["sum"] = torch.empty(3, dtype=s["q"].dtype, device="cuda"), s["q"].new_empty(1)
    return s


def run(state):
    c = state["case"]
    k = c["kind"]
    if k == "step":
        m = state["m"]
        m.restore_snapshot()
        m.step_async(c["dt"], 6, c["steps"])
        with torch.cuda.stream(state["stream"]):
            return fields_of(m, range(12 if c["moist"] else 7), c["mixed"])
    if k == "nested":
        state["n"].wait()  # the members are the set's until its launched steps are done
        for m in state["models"]:
            m.restore_snapshot()
            m.sync()
        state["n"].step_async(18.0, 6, 1)
        with torch.cuda.stream(state["stream"]):
            return [fields_of(m, range(7), True) for m in state["models"]]
    if k == "helmholtz":
        state["h"].solve_dev(state["f"].data_ptr(), state["x"].data_ptr(), torch.cuda.current_stream().cuda_stream)
        return state["x"]
    if k == "window":
        w = state["w"]
        out = w.ad(state["pert"]) if c["adjoint"] else w.tl(state["pert"])
        s = state["m"].setup
        out = [vg.interior(s, sp, out[sp]) for sp in range(7)]
        return [a.astype(np.float32) for a in out] if c["mixed"] else out
    st = torch.cuda.current_stream().cuda_stream
    t = "f64" if c["f64"] else "f32"
    if k == "columns":
        _ok(_c["tridiagonal_solve_batched", t](state["a"].data_ptr(), state["b"].data_ptr(), state["c"].data_ptr(),
                                               state["d"].data_ptr(), c["n"], c["systems"], state["x"].data_ptr(),
                                               None, st))
        return state["x"]
    zs = state["zs"].data_ptr() if state["zs"] is not None else None
    if k == "flux":
        _ok(_c["advect_scalar_flux", t](*[state[f].data_ptr() for f in ("q", "rho", "u", "v", "w", "dzeta")], zs,
                                        c["nx"], c["ny"], c["nz"], 1000.0, 1000.0, 20000.0, state["out"].data_ptr(),
                                        st))
        return state["out"]
    _ok(_c["cfl_scan", t](*[state[f].data_ptr() for f in ("u", "v", "w", "dzeta")], zs, c["nx"], c["ny"], c["nz"],
                          1000.0, 1000.0, 20000.0, 6.0, state["cfl"].data_ptr(), st))
    _ok(_c["neumaier_sum", t](state["rho"].data_ptr(), cells_of(c), state["sum"].data_ptr(), st))
    return state["cfl"], state["sum"]


def work(case):
    """Inputs read once, outputs written once; arithmetic per cell counted
    from the formulas (about 3400 flops per cell of a dry step: 3 x 830 for a
    slow tendency, 18 x 50 for the substeps)."""
    k = case["kind"]
    if k == "step":
        n, sp = cells_of(case), 12 if case["moist"] else 7
        out = 4 if case["mixed"] else 8
        return dict(bytes=n * sp * (8 + out), flops=n * case["steps"] * (9000 if case["moist"] else 3400))
    if k == "nested":
        p = cells_of(case)
        ch = sum(nx * ny for nx, ny, _, _ in nest_boxes(case)) * case["nz"]
        return dict(bytes=(p + ch) * 7 * 12, flops=3400 * (p + 3 * ch))
    if k == "helmholtz":
        return dict(bytes=cells_of(case) * 8 * 4, flops=cells_of(case) * 1500)
    if k == "window":
        n = cells_of(case)
        # trajectory plus linear sweep; the adjoint recomputes its trajectory
        return dict(bytes=n * 7 * 24, flops=n * case["steps"] * (17000 if case["adjoint"] else 10000))
    size = 8 if case["f64"] else 4
    if k == "columns":
        n = case["n"] * case["systems"]
        return dict(bytes=size * 5 * n, flops=9 * n)
    n = cells_of(case)
    return dict(bytes=size * (6 if k == "flux" else 4) * n, flops=n * (40 if k == "flux" else 20))


# ---- the same results from plain torch in 64 bits ----
def _at(f, axis, idx, top=None):
    """f at the indices idx along axis, clamped to 0..top (its last cell)."""
    top = f.shape[axis] - 1 if top is None else top
    return f.index_select(axis, torch.as_tensor(idx, device=f.device).clamp(0, top))


def _weno_left(a, b, c, d, e):
    v0, v1, v2 = (2 * a - 7 * b + 11 * c) / 6, (-b + 5 * c + 2 * d) / 6, (2 * c + 5 * d - e) / 6
    s0 = 13 / 12 * (a - 2 * b + c) ** 2 + 0.25 * (a - 4 * b + 3 * c) ** 2
    s1 = 13 / 12 * (b - 2 * c + d) ** 2 + 0.25 * (b - d) ** 2
    s2 = 13 / 12 * (c - 2 * d + e) ** 2 + 0.25 * (3 * c - 4 * d + e) ** 2
    w0, w1, w2 = 0.1 / (1e-6 + s0) ** 2, 0.6 / (1e-6 + s1) ** 2, 0.3 / (1e-6 + s2) ** 2
    return (w0 * v0 + w1 * v1 + w2 * v2) / (w0 + w1 + w2)


def _face_flux(q, vel, axis):
    n = q.shape[axis]
    f = torch.arange(n + 1, device=q.device)
    z = [_at(q, axis, f + o) for o in (-3, -2, -1, 0, 1)]
    ql, qr = _weno_left(*z), _weno_left(*z[::-1])
    al = torch.where(vel >= 1e-3, vel, torch.where(vel <= -1e-3, -vel, torch.full_like(vel, 1e-3)))
    return 0.5 * (vel * (ql + qr) - al * (qr - ql))


class _Step:
    """The dry step of ``setup_of`` in plain torch operations."""

    def __init__(self, nx, ny, nz, dx, z_top, beta, rigid):
        zeta = zeta_of(nz)
        th0, pi0, rho0 = base_of(zeta, z_top)
        col = lambda a: torch.tensor(a, dtype=F64, device="cuda")[:, None, None]  # noqa: E731
        self.th0, self.pi0, self.rho0 = col(th0), col(pi0), col(rho0)
        dz = np.maximum(np.diff(zeta) * z_top, 1.0)
        kc, km = np.minimum(np.arange(nz + 1), nz - 1), np.maximum(np.arange(nz + 1) - 1, 0)
        self.dz, self.dzf = col(dz), col(dz[kc])
        self.rf, self.tf = col(0.5 * (rho0[km] + rho0[kc])), col(0.5 * (th0[km] + th0[kc]))
        self.kap = col(RD / CV * pi0 / rho0)
        zc = 0.5 * (zeta[:-1] + zeta[1:]) * z_top
        t = np.clip((zc - 0.8 * z_top) / (0.2 * z_top), 0.0, 1.0)
        self.sponge = np.where(zc > 0.8 * z_top, 0.2 * np.sin(0.5 * math.pi * t) ** 2, 0.0)
        self.kc = kc
        self.T = 0.5 * (rho0[km] + rho0[kc]) * CP * 0.5 * (th0[km] + th0[kc]) / dz[kc]
        self.T[0] = self.T[nz] = 0.0
        self.c = RD / CV * pi0 / rho0 / dz
        self.nx, self.ny, self.nz, self.dx, self.beta, self.rigid = nx, ny, nz, dx, beta, rigid

    def slow(self, u, v, w, rho, th, pi):
        nx, ny, nz, dx = self.nx, self.ny, self.nz, self.dx
        dev = u.device
        i0, i1 = torch.arange(nx, device=dev), torch.arange(nx + 1, device=dev)
        j0, j1 = torch.arange(ny, device=dev), torch.arange(ny + 1, device=dev)
        k0, k1 = torch.arange(nz, device=dev), torch.arange(nz + 1, device=dev)
        X, Y, Z = 2, 1, 0
        tp, pp = th - self.th0, pi - self.pi0
        # u faces
        um, up = _at(u, X, i1 - 1, nx - 1), _at(u, X, i1, nx - 1)
        vm, vp = _at(v, Y, j0 - 1), _at(v, Y, j0)
        vs = vm + vp
        vc = 0.25 * (_at(vs, X, i1 - 1) + _at(vs, X, i1))
        ws = 0.5 * (_at(w, Z, k0) + _at(w, Z, k0 + 1, nz - 1))
        du = -(0.5 * (um + up) * (up - um) / dx + vc * (_at(up, Y, j0 + 1) - _at(up, Y, j0 - 1)) / (2 * dx) +
               _at(ws, X, i1) * (_at(up, Z, k0 + 1) - _at(up, Z, k0 - 1)) / (2 * self.dz))
        du = du - CP * 0.5 * (_at(tp, X, i1 - 1) + _at(tp, X, i1)) * (_at(pp, X, i1) - _at(pp, X, i1 - 1)) / dx
        # v faces
        vm, vp = _at(v, Y, j1 - 1, ny - 1), _at(v, Y, j1, ny - 1)
        us = _at(u, X, i0 - 1) + _at(u, X, i0)
        uc = 0.25 * (_at(us, Y, j1 - 1) + _at(us, Y, j1))
        dv = -(uc * (_at(vp, X, i0 + 1) - _at(vp, X, i0 - 1)) / (2 * dx) + 0.5 * (vm + vp) * (vp - vm) / dx +
               _at(ws, Y, j1) * (_at(vp, Z, k0 + 1) - _at(vp, Z, k0 - 1)) / (2 * self.dz))
        dv = dv - CP * 0.5 * (_at(tp, Y, j1 - 1) + _at(tp, Y, j1)) * (_at(pp, Y, j1) - _at(pp, Y, j1 - 1)) / dx
        # w faces
        wk, wm = w, _at(w, Z, k1 - 1)
        uc = 0.5 * (_at(u, X, i0) + _at(u, X, i0 + 1))
        vc = 0.5 * (_at(v, Y, j0) + _at(v, Y, j0 + 1))
        dw = -(_at(uc, Z, k1) * (_at(wk, X, i0 + 1) - _at(wk, X, i0 - 1)) / (2 * dx) +
               _at(vc, Z, k1) * (_at(wk, Y, j0 + 1) - _at(wk, Y, j0 - 1)) / (2 * dx) +
               0.5 * (_at(w, Z, k1, nz - 1) + wk) * (wk - wm) / self.dzf)
        dw = dw - CP * 0.5 * (_at(tp, Z, k1 - 1) + _at(tp, Z, k1)) * (_at(pp, Z, k1) - _at(pp, Z, k1 - 1)) / self.dzf
        dw = dw + G * _at(tp / self.th0, Z, k1)
        # mass: the full flux minus its linear part; rho is 0 beyond the domain
        def halves(f, axis, n):
            e = torch.zeros_like(f.narrow(axis, 0, 1))
            lo = torch.cat([f.narrow(axis, 0, 1), f], axis)
            hi = torch.cat([f, e], axis)
            return 0.5 * (lo + hi)
        rx = halves(rho, X, nx) - self.rho0
        ry = halves(rho, Y, ny) - self.rho0
        rz = 0.5 * (_at(rho, Z, k1 - 1) + _at(rho, Z, k1)) - self.rf
        dr = -(torch.diff(u * rx, dim=X) / dx + torch.diff(v * ry, dim=Y) / dx +
               torch.diff(w * rz, dim=Z) / self.dz)
        div = torch.diff(u, dim=X) / dx + torch.diff(v, dim=Y) / dx + torch.diff(w, dim=Z) / self.dz
        dth = -(torch.diff(_face_flux(th, u, X), dim=X) / dx + torch.diff(_face_flux(th, v, Y), dim=Y) / dx +
                torch.diff(_face_flux(th, w, Z), dim=Z) / self.dz) + th * div
        return du, dv, dw, dr, dth

    def substep(self, u, v, w, rho, pi, dtau):
        nz, dx, b = self.nz, self.dx, self.beta
        ob = 1.0 - b
        dh = -self.rho0 * (torch.diff(u, dim=2) + torch.diff(v, dim=1)) / dx
        pp = pi - self.pi0
        zero = torch.zeros_like(pp[:1])
        grad = lambda x: torch.cat([zero, (x[1:] - x[:-1]) / self.dzf[1:nz], zero])  # noqa: E731
        dvz = lambda f: -torch.diff(self.rf * f, dim=0) / self.dz  # noqa: E731
        wt = w - dtau * ob * CP * self.tf * grad(pp)
        old = dvz(w)
        rhs = pp + dtau * self.kap * (dh + ob * old + b * dvz(wt))
        T, ck = self.T.tolist(), ((dtau * b) ** 2 * self.c).tolist()
        cp, dp = [], []
        for k in range(nz):
            lo, up, dg = -ck[k] * T[k], -ck[k] * T[k + 1], 1.0 + ck[k] * (T[k] + T[k + 1])
            den = dg - lo * cp[-1] if k else dg
            dp.append((rhs[k] - lo * dp[-1]) / den if k else rhs[k] / den)
            cp.append(up / den)
        x = [dp[-1]]
        for k in range(nz - 2, -1, -1):
            x.append(dp[k] - cp[k] * x[-1])
        x = torch.stack(x[::-1])
        w = wt - dtau * b * CP * self.tf * grad(x)
        rho = rho + dtau * (dh + ob * old + b * dvz(w))
        gx = torch.nn.functional.pad(torch.diff(x, dim=2), (1, 1)) / dx
        gy = torch.nn.functional.pad(torch.diff(x, dim=1), (0, 0, 1, 1)) / dx
        return u - dtau * CP * self.th0 * gx, v - dtau * CP * self.th0 * gy, w, rho, x + self.pi0

    def __call__(self, dt, n_sub, u, v, w, rho, th, pi):
        s = (u, v, w, rho, th)
        cur = s + (pi,)
        for h in (dt / 3, dt / 2, dt):
            d = self.slow(*cur)
            a, b, c, r, t = (f + h * g for f, g in zip(s, d))
            p = pi
            for _ in range(n_sub):
                a, b, c, r, p = self.substep(a, b, c, r, p, h / n_sub)
            cur = (a, b, c, r, t, p)
        a, b, c, r, t, p = cur
        al = torch.tensor(self.sponge, dtype=F64, device="cuda")[:, None, None]
        k = 1.0 / (1.0 + dt * al)
        kw = k[torch.as_tensor(self.kc, device="cuda")]
        c = c * kw
        if self.rigid:
            c = torch.nn.functional.pad(c[1:-1], (0, 0, 0, 0, 1, 1))
        r, t, p = (k * (f + dt * al * f0) for f, f0 in ((r, self.rho0), (t, self.th0), (p, self.pi0)))
        return a * k, b * k, c, r, t, p


def _exact_helmholtz(case, seed):
    dz, zs, a, b, f = hill_inputs(case, seed)
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    h = torch.tensor(dz, dtype=F64, device="cuda")[:, None, None] * \
        (20000.0 - torch.tensor(zs, dtype=F64, device="cuda"))[None]
    D2 = 4e6

    def face(axis, m):
        lo = 0.5 * (a.narrow(axis, 1, m - 1) + a.narrow(axis, 0, m - 1))
        pad = [0, 0, 0, 0, 0, 0]
        pad[2 * (2 - axis)] = pad[2 * (2 - axis) + 1] = 1
        return torch.nn.functional.pad(lo, pad), pad

    (ax, px), (ay, py), (az, pz) = face(2, nx), face(1, ny), face(0, nz)

    def apply(x):
        gx = ax * torch.nn.functional.pad(torch.diff(x, dim=2), px)
        gy = ay * torch.nn.functional.pad(torch.diff(x, dim=1), py)
        gz = az * torch.nn.functional.pad(torch.diff(x, dim=0), pz)
        return b * x - torch.diff(gx, dim=2) / D2 - torch.diff(gy, dim=1) / D2 - torch.diff(gz, dim=0) / (h * h)

    # Jacobi in the horizontal, the exact tridiagonal in the vertical
    dg = b + (ax[:, :, 1:] + ax[:, :, :-1] + ay[:, 1:] + ay[:, :-1]) / D2 + (az[1:] + az[:-1]) / (h * h)
    lo, up = -az[:-1] / (h * h), -az[1:] / (h * h)
    cp, inv = [], []
    for k in range(nz):
        inv.append(1.0 / (dg[k] - lo[k] * cp[-1] if k else dg[k]))
        cp.append(up[k] * inv[k])

    def precond(r):
        y = []
        for k in range(nz):
            y.append((r[k] - lo[k] * y[-1] if k else r[k]) * inv[k])
        for k in range(nz - 2, -1, -1):
            y[k] = y[k] - cp[k] * y[k + 1]
        return torch.stack(y)

    dot = lambda p, q: (p * q).sum()  # noqa: E731
    x = torch.zeros_like(f)
    fn = f.norm()
    for _ in range(4):  # restarted from the true residual
        r = f - apply(x)
        r0, rho, al, om = r.clone(), torch.ones((), dtype=F64, device="cuda"), 1.0, 1.0
        v = p = torch.zeros_like(f)
        for it in range(300):
            rn = dot(r0, r)
            p = r + (rn / rho) * (al / om) * (p - om * v)
            rho = rn
            ph = precond(p)
            v = apply(ph)
            al = rho / dot(r0, v)
            s = r - al * v
            sh = precond(s)
            t = apply(sh)
            om = dot(t, s) / dot(t, t)
            x = x + al * ph + om * sh
            r = s - om * t
            if it % 8 == 7 and float(r.norm() / fn) < 2e-14:
                break
        if float((f - apply(x)).norm() / fn) < 1e-13:
            break
    return x


def exact(case, seed):
    k = case["kind"]
    if k == "step":
        if case["moist"]:  # the warm-rain scheme is not restated here
            return None
        m = _Step(case["nx"], case["ny"], case["nz"], case["dx"], case["z_top"], 0.5, 0)
        s = member(case["nx"], case["ny"], case["nz"], case["dx"], case["z_top"], seed)
        cur = tuple(s[:6])
        for _ in range(case["steps"]):
            cur = m(case["dt"], 6, *cur)
        return list(cur) + [s[QV]]
    if k == "nested":  # one long chain of the other cases' steps and transfers
        return None
    if k == "helmholtz":
        return _exact_helmholtz(case, seed)
    if k == "window":
        m = _Step(case["nx"], case["ny"], case["nz"], WIN["dx"], WIN["z_top"], WIN["beta"], WIN["rigid"])
        state, pert = window_inputs(case, seed)

        def model(*s):
            for _ in range(case["steps"]):
                s = m(WIN["dt"], 6, *s)
            return s

        if case["adjoint"]:
            xs = [f.clone().requires_grad_(True) for f in state[:6]]
            out = list(torch.autograd.grad(model(*xs), xs, pert[:6]))
        else:
            out = list(torch.func.jvp(model, tuple(state[:6]), tuple(pert[:6]))[1])
        # qv = 0: the adjoint sees it through the buoyancy, as the model's does
        return out + [None if case["adjoint"] else torch.zeros_like(state[QV])]
    if k == "columns":
        a, b, c, d = (t.double() for t in column_inputs(case, seed))
        cp, dp = torch.empty_like(b), torch.empty_like(b)
        for i in range(case["n"]):
            den = b[:, i] - a[:, i - 1] * cp[:, i - 1] if i else b[:, 0]
            dp[:, i] = (d[:, i] - a[:, i - 1] * dp[:, i - 1]) / den if i else d[:, 0] / den
            cp[:, i] = c[:, i] / den if i + 1 < case["n"] else 0.0
        for i in range(case["n"] - 2, -1, -1):
            dp[:, i] -= cp[:, i] * dp[:, i + 1]
        return dp
    s = {f: None if t is None else t.double() for f, t in grid_inputs(case, seed).items()}
    depth = 20000.0 - (s["zs"] if s["zs"] is not None else 0.0)
    dz = torch.clamp(s["dzeta"][:, None, None] * depth, min=1.0)
    if k == "flux":
        q, r = s["q"], s["rho"]

        def west(f, axis):
            return f * 0.25 * (r + r.roll(1, axis)) * (q + q.roll(1, axis))

        fx, fy, fz = west(s["u"], 2), west(s["v"], 1), west(s["w"], 0)
        div = (fx.roll(-1, 2) - fx) / 1000.0 + (fy.roll(-1, 1) - fy) / 1000.0
        div[1:-1] += ((fz.roll(-1, 0) - fz) / dz)[1:-1]
        return -div / r.clamp(min=1e-12)
    u, v, w = s["u"], s["v"], s["w"]
    cfl = 6.0 * (u.abs() / 1000.0 + v.abs() / 1000.0 + w.abs() / dz)
    top = torch.stack([cfl.max(), (u * u + v * v + w * w).max().sqrt(), dz.min()])
    return top, s["rho"].sum().reshape(1)
