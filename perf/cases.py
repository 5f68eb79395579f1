"""Work a user has this library do, as cases with sizes, inputs and outputs.

Kinds of case:

* ``vortcor``: the allocation-free vorticity correction on device arrays that
  the caller owns;
* ``par2grid``: one par2grid of parcels in container order, the fields read
  back (a host code that calls the step's procedures one by one);
* ``host``: the drop-in step of a host that owns the parcel container: parcels
  in, one step, parcels out;
* ``restart``: deformed parcels of a developed flow loaded, some steps, the
  fields read back;
* ``run``: an initial state generated on the device (rising thermal or Beltrami
  flow), some steps, the fields read back (what a served request does).

Grids, domains, options and flows are those of the package's workloads
(epic_b200.initial, the served ensemble, the parity tests); the grids with
other factors stand for a user's own.
"""
import ctypes as C
import math

import numpy as np
import torch

import epic_b200
from epic_b200 import abi
from epic_b200.serve import beltrami_zeta_flags

# fields a run writes out: vorticity, velocity, total and dry buoyancy, humidity, volume
FIELDS = abi.VORTG + abi.VELOG + (abi.TBUOYG, abi.DBUOYG, abi.HUMG, abi.VOLG)
# what par2grid computes
P2G_FIELDS = abi.VORTG + (abi.TBUOYG, abi.DBUOYG, abi.HUMG, abi.VOLG, abi.NPARG, abi.NSPARG)


def _run(name, flow, nx, ny, nz, precision, steps, keep_order=0):
    return dict(name=name, kind="run", flow=flow, nx=nx, ny=ny, nz=nz, precision=precision, steps=steps,
                keep_order=keep_order)


def _restart(name, nx, ny, nz, precision, steps):
    return dict(name=name, kind="restart", nx=nx, ny=ny, nz=nz, precision=precision, steps=steps, keep_order=0)


def listed():
    return [
        # the smallest call: a correction inside another code's time loop
        dict(name="vortcor-200003", kind="vortcor", n=200003),
        # a small host-owned container, an odd number of cells along z
        dict(name="host-24x20x17-fp64", kind="host", nx=24, ny=20, nz=17, precision=0, keep_order=0),
        # par2grid on its own; axes that are not powers of two
        dict(name="par2grid-40x60x36-fp64", kind="par2grid", nx=40, ny=60, nz=36, precision=0, keep_order=1),
        dict(name="par2grid-64-mixed", kind="par2grid", nx=64, ny=64, nz=64, precision=1, keep_order=1),
        # the reference's CPU configuration
        _run("beltrami-32-fp64", "beltrami", 32, 32, 32, 0, 10),
        # two of the served ensemble's requests
        _run("thermal-48-mixed", "thermal", 48, 48, 48, 1, 10),
        _run("beltrami-96x96x48-mixed", "beltrami", 96, 96, 48, 1, 6),
        # developed flows: parcels deformed up to the split threshold, some small
        _restart("restart-64-fp64", 64, 64, 64, 0, 4),
        _restart("restart-80x72x60-mixed", 80, 72, 60, 1, 4),
        # the default store order of the C interface
        _run("thermal-64-kept-order-fp64", "thermal", 64, 64, 64, 0, 4, keep_order=1),
        # the headline workload and the mixed form's own
        _run("thermal-128-fp64", "thermal", 128, 128, 128, 0, 3),
        _run("thermal-256x256x128-mixed", "thermal", 256, 256, 128, 1, 2),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


_AXES = (16, 18, 20, 24, 30, 32, 36, 40, 48, 54, 60, 64, 72, 80, 90, 96, 100, 108, 120, 128)


def _grid(rng, most):
    """Even x and y axes with factors 2, 3, 5 and any z axis, at most `most` cells."""
    while True:
        nx, ny = rng.choice(_AXES), rng.choice(_AXES)
        nz = round(_log(rng, 12, 128))
        if nx <= 3 * ny and ny <= 3 * nx and nz <= 3 * max(nx, ny) and nx * ny * nz <= most:
            return nx, ny, nz


def draw(rng):
    kind = rng.choice(("vortcor", "host", "par2grid", "restart", "restart", "run", "run", "run"))
    if kind == "vortcor":
        return dict(kind=kind, n=round(_log(rng, 1000, 4e6)))
    if kind == "host":
        nx, ny, nz = _grid(rng, 64 ** 3)
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, precision=0, keep_order=rng.randrange(2))
    if kind == "par2grid":
        nx, ny, nz = _grid(rng, 64 ** 3)
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, precision=rng.randrange(2), keep_order=rng.randrange(2))
    nx, ny, nz = _grid(rng, 96 ** 3)
    steps = rng.randint(2, 6)
    if kind == "restart":
        return dict(kind=kind, nx=nx, ny=ny, nz=nz, precision=rng.randrange(2), steps=steps, keep_order=rng.randrange(2))
    return dict(kind=kind, flow=rng.choice(("thermal", "beltrami")), nx=nx, ny=ny, nz=nz,
                precision=rng.randrange(2), steps=steps, keep_order=int(rng.random() < 0.3))


# ---------------------------------------------------------------------------
# inputs

def _mode(seed):
    """A Beltrami state has no random part: the seed picks its wave numbers."""
    return 1 + seed % 3, 1 + seed // 3 % 3, 1 + seed // 9 % 2


def _domain(case, seed):
    """(lower, extent, options) of the case's flow."""
    if case.get("flow") == "beltrami":
        flags = beltrami_zeta_flags((case["nx"], case["ny"], case["nz"]), _mode(seed))
        return ((-math.pi, -math.pi, -0.5 * math.pi), (2 * math.pi, 2 * math.pi, math.pi),
                dict(min_vratio=40.0, lambda_max=4.0, bndry_zeta_zero=flags))
    # cells are nearly cubes, as in the package's workloads
    h = 6.28 / max(case["nx"], case["ny"])
    ext = (h * case["nx"], h * case["ny"], h * case["nz"])
    return ((-0.5 * ext[0], -0.5 * ext[1], 0.0), ext,
            dict(min_vratio=40.0, lambda_max=4.0, bndry_zeta_zero=(0, 0)))


def _parcels(case, seed):
    """Parcels of a developed flow, 8 per cell, made on the GPU in container
    order: displaced from the regular positions by up to 0.9 of their spacing,
    aspect ratios up to just above the split threshold, volumes over a factor
    of three with one in a hundred below the merge threshold, a smooth
    vorticity field with parcel noise, warm moist air in the middle.  The host's
    container is calmer (nothing splits or merges within the step), so that its
    size stays."""
    calm = case["kind"] == "host"
    lower, ext, opts = _domain(case, seed)
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    dx = [ext[0] / nx, ext[1] / ny, ext[2] / nz]
    g = torch.Generator(device="cuda").manual_seed(seed)
    dev = dict(dtype=torch.float64, device="cuda")

    def rnd(*shape):
        return torch.rand(*shape, generator=g, **dev)

    n = nx * ny * nz * 8
    i = torch.arange(n, device="cuda")
    sub, cell = i % 8, i // 8
    at = [(cell % nx) * 2 + sub % 2, (cell // nx % ny) * 2 + sub // 2 % 2, (cell // (nx * ny)) * 2 + sub // 4]
    pos = torch.empty(n, 3, **dev)
    for k in range(3):
        x = lower[k] + (at[k] + 0.5 + 0.9 * (2 * rnd(n) - 1)) * (0.5 * dx[k])
        if k < 2:
            x = lower[k] + (x - lower[k]) % ext[k]
        else:
            x = x.clamp(lower[k], lower[k] + ext[k] * (1 - 1e-12))
        pos[:, k] = x
    vcell = dx[0] * dx[1] * dx[2]
    vol = torch.exp(math.log(1.5 if calm else 3.0) * (rnd(n) - 0.5))
    small = rnd(n) < (0.0 if calm else 0.01)
    vol = torch.where(small, 0.15 * vol, vol)
    vol *= vcell * nx * ny * nz / vol.sum()
    # B = R diag(a^2, b^2, c^2) R^T with a b c = 3 vol / 4 pi
    ratio = torch.exp(math.log(1.5 if calm else 4.02) * torch.sqrt(rnd(n)))       # a / c
    mid = torch.exp(torch.log(ratio) * rnd(n))                     # b / c
    c2 = (0.75 * vol / math.pi / (ratio * mid)) ** (2.0 / 3.0)
    ax = torch.stack([ratio ** 2 * c2, mid ** 2 * c2, c2], 1)
    q = torch.randn(n, 4, generator=g, **dev)
    q /= q.norm(dim=1, keepdim=True)
    w, x, y, z = q.unbind(1)
    R = torch.stack([1 - 2 * (y * y + z * z), 2 * (x * y - w * z), 2 * (x * z + w * y),
                     2 * (x * y + w * z), 1 - 2 * (x * x + z * z), 2 * (y * z - w * x),
                     2 * (x * z - w * y), 2 * (y * z + w * x), 1 - 2 * (x * x + y * y)], 1).view(n, 3, 3)

    def b(r, s):
        return (R[:, r] * R[:, s] * ax).sum(1)

    B = torch.stack([b(0, 0), b(0, 1), b(0, 2), b(1, 1), b(1, 2)], 1)
    th = [2 * math.pi * (pos[:, k] - lower[k]) / ext[k] for k in range(3)]
    ph = 2 * math.pi * torch.rand(3, generator=g, **dev)
    vor = torch.stack([torch.sin(th[1] + ph[0]) * torch.cos(0.5 * th[2]), torch.sin(th[0] + ph[1]) * torch.cos(0.5 * th[2]),
                       torch.sin(th[0] + th[1] + ph[2]) * torch.sin(0.5 * th[2])], 1)
    vor += 0.05 * torch.randn(n, 3, generator=g, **dev)
    r2 = ((pos - torch.tensor([lower[k] + 0.5 * ext[k] for k in range(3)], **dev)) ** 2).sum(1) / (0.3 * min(ext)) ** 2
    buoy = 0.5 * torch.exp(-r2) + 1e-3 * (2 * rnd(n) - 1)
    hum = 0.016 * torch.exp(-r2) * (0.9 + 0.1 * rnd(n))
    return (lower, ext, opts), (pos, vor, B, vol, buoy, hum)


class _State:
    """A context, what a pass takes into it and the pinned arrays it reads into."""

    def __init__(self, case, domain, fields=()):
        self.case = case
        self.lib = epic_b200.load()
        lower, ext, opts = domain
        n = case["nx"] * case["ny"] * case["nz"] * 8
        cfg = self.lib.default_config(case["nx"], case["ny"], case["nz"], lower, ext, precision=case["precision"],
                                      keep_order=case["keep_order"],
                                      # the default (twice the parcels at the start), less for the largest
                                      capacity=0 if n < 20e6 else int(1.3 * n), **opts)
        self.ctx = epic_b200.EpicContext(self.lib, cfg)
        self.fields = fields
        self.out = {f: torch.empty(self.ctx.field_shape, dtype=torch.float64, pin_memory=True) for f in fields}

    def read_fields(self):
        for f, a in self.out.items():
            self.ctx._call("get_field", C.c_int(f), _ptr(a))
        return {abi.FIELD_NAMES[f]: a for f, a in self.out.items()}

    def load(self):
        pos, vor, B, vol, buoy, hum = self.host
        self.ctx._call("set_parcels", C.c_int64(len(vol)), _ptr(pos), _ptr(vor), _ptr(B), _ptr(vol), _ptr(buoy), _ptr(hum))


def _ptr(t):
    return C.cast(t.data_ptr(), C.POINTER(C.c_double))


def _pinned(t):
    h = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    h.copy_(t)
    return h


def prepare(case, seed):
    kind = case["kind"]
    if kind == "vortcor":
        g = torch.Generator(device="cuda").manual_seed(seed)
        n = case["n"]
        vol = 0.5 + torch.rand(n, generator=g, dtype=torch.float64, device="cuda")
        vor = 0.3 + torch.randn(n, 3, generator=g, dtype=torch.float64, device="cuda")
        f = epic_b200.load().lib.epic_gpu_apply_vortcor_noalloc
        f.argtypes = [C.c_int64, C.c_void_p, C.c_void_p, C.POINTER(C.c_double), C.POINTER(C.c_double), C.c_void_p]
        f.restype = C.c_int
        torch.cuda.synchronize()
        return dict(kind=kind, n=n, vol=vol, vor=vor, call=f, vbar=(C.c_double * 3)(0.1, -0.2, 0.05))
    if kind == "run":
        s = _State(case, _domain(case, seed), FIELDS)
        if case["flow"] == "thermal":
            lower, ext = s.ctx.cfg.lower, s.ctx.cfg.extent
            s.spec = abi.init_spec(abi.INIT_THERMAL, 8, seed, bubbles=((0.0, 0.0, lower[2] + 0.25 * ext[2], 0.5),))
        else:
            s.spec = abi.init_spec(abi.INIT_BELTRAMI, 8, seed, klm=_mode(seed))
        return s
    domain, parcels = _parcels(case, seed)
    s = _State(case, domain, {"par2grid": P2G_FIELDS, "restart": FIELDS, "host": ()}[kind])
    s.host = [_pinned(t) for t in parcels]
    if kind == "par2grid":
        s.load()
    if kind == "host":
        n, cap = len(s.host[3]), int(2 * len(s.host[3])) + 1024
        s.back = [torch.empty((cap,) + tuple(t.shape[1:]), dtype=torch.float64, pin_memory=True) for t in s.host]
    return s


def _steps(s, count):
    t, info, dts = 0.0, None, []
    for _ in range(count):
        t, info = s.ctx.step(t)
        dts.append(info.dt)
    counts = [info.n_parcels, info.n_splits, info.n_merges]
    # the mixed form's split and merge decisions follow its FP32 shapes
    out = dict(time=np.array([t] + dts), counts=np.array(counts, dtype=np.float64 if s.case["precision"] else np.int64),
               parcel_stats=np.array(info.parcel_stats), field_stats=np.array(info.field_stats))
    return out


def run(s):
    if isinstance(s, dict):
        rc = s["call"](s["n"], s["vol"].data_ptr(), s["vor"].data_ptr(), s["vbar"], None, None)
        assert rc == 0, rc
        return s["vor"]
    kind = s.case["kind"]
    if kind == "par2grid":
        s.ctx.par2grid(False)
        return s.read_fields()
    if kind == "run":
        s.ctx.init_state(s.spec)
        s.ctx.init_correction()
        out = _steps(s, s.case["steps"])
        out.update(s.read_fields())
        return out
    s.load()
    s.ctx.init_correction()
    if kind == "restart":
        out = _steps(s, s.case["steps"])
        out.update(s.read_fields())
        return out
    out = _steps(s, 1)
    n = C.c_int64()
    s.ctx._call("get_parcels", C.c_int64(len(s.back[3])), C.byref(n), *(_ptr(t) for t in s.back))
    out.update(zip(("pos", "vor", "B", "vol", "buoy", "hum"), (t[:n.value] for t in s.back)))
    return out


# ---------------------------------------------------------------------------
# what a pass cannot do without

def work(case):
    if case["kind"] == "vortcor":
        # volume twice (sum, correction), vorticity in and out; the sums of the correction
        return {"bytes": case["n"] * 8 * 7, "flops": case["n"] * 10}
    cells = case["nx"] * case["ny"] * case["nz"]
    n = cells * 8
    grid = case["nx"] * case["ny"] * (case["nz"] + 3) * 8
    e = 4 if case["precision"] else 8
    state = 4 * 8 + 10 * e                       # position, volume; vorticity, B, buoyancy, humidity
    # support points and weights, 4 points x 8 corners x 7 fields
    p2g_flops = n * (150 + 4 * (30 + 8 * 7 * 2))
    if case["kind"] == "par2grid":
        return {"bytes": n * state + 7 * grid, "flops": p2g_flops}
    # per stage: par2grid and grid2par each read position, support vectors and
    # their attributes once, and the update reads and writes the state and the
    # accumulators; four vol2grids and moves, split and merge tests
    stage = (3 * 8 + 6 * e + 8 + 5 * e) + 2 * (6 * 8 + 16 * e) + 8 + 6 * e
    per_step = n * (5 * stage + 4 * (8 * 7 + 6 * e) + 2 * state + 8 + 5 * e) + 5 * 45 * grid
    flops = 5 * (p2g_flops + n * (4 * (30 + 8 * 14 * 2) + 200)) + 4 * n * 4 * 60
    steps = case.get("steps", 1)
    return {"bytes": steps * per_step + (n * 2 * state if case["kind"] != "run" else n * state), "flops": steps * flops}


def tolerance(case):
    # about four times what other FFT kernels, the other store order, FP64
    # spectral work in the mixed form and (par2grid) 64-bit sums change
    if case["kind"] == "vortcor":
        return {"rel": 1e-14}
    if case["kind"] == "par2grid":
        return {"rel": 8e-7, "max": 4e-5} if case["precision"] else {"rel": 1.5e-13, "max": 1e-11}
    if case.get("flow") == "thermal":
        # vertical vorticity is still far below the other components
        return {"rel": 2.8e-3, "max": 0.12} if case["precision"] else {"rel": 6e-12, "max": 2.6e-10}
    # a split or merge decision at its threshold moves a mixed run's volumes there
    return {"rel": 4e-6, "max": 1e-2} if case["precision"] else {"rel": 2e-13, "max": 4e-12}


# ---------------------------------------------------------------------------
# the same in 64 bits

def _support_points(pos, B, vol):
    abc = 0.75 * vol / math.pi
    b11, b12, b13, b22, b23 = B.unbind(1)
    b33 = (abc ** 2 - b13 * (b12 * b23 - b13 * b22) + b11 * b23 ** 2 - b12 * b13 * b23) / (b11 * b22 - b12 ** 2)
    U = torch.stack([b11, b12, b13, b12, b22, b23, b13, b23, b33], 1).view(-1, 3, 3)
    parts = [torch.linalg.eigh(u) for u in U.split(10000)]
    D = torch.cat([p[0] for p in parts])            # ascending
    V = torch.cat([p[1] for p in parts])
    eta = torch.sqrt((D[:, 2] - D[:, 0]).abs() * 0.4)[:, None] * V[:, :, 2]
    tau = torch.sqrt((D[:, 1] - D[:, 0]).abs() * 0.4)[:, None] * V[:, :, 1]
    r = math.sqrt(0.5)
    return [pos + r * (s * eta + t * tau) for s in (1, -1) for t in (1, -1)]


def exact(case, seed):
    if case["kind"] == "vortcor":
        s = prepare(case, seed)
        vol, vor = s["vol"], s["vor"]
        mean = (vor * vol[:, None]).sum(0) / vol.sum()
        return vor - (mean - torch.tensor(list(s["vbar"]), dtype=torch.float64, device="cuda"))
    if case["kind"] != "par2grid":
        return None   # whole steps: no plain program of 20 seconds computes them
    (lower, ext, opts), (pos, vor, B, vol, buoy, hum) = _parcels(case, seed)
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    dxi = [nx / ext[0], ny / ext[1], nz / ext[2]]
    # latent heat and the saturation profile of the default physics
    glat = 9.80616 * float(np.float32(2.501e6)) / (1005.7 * 288.15)
    qc = (hum - 0.015 * torch.exp((lower[2] - pos[:, 2]) / 1000.0)).clamp(min=0.0)
    vals = dict(x=vor[:, 0], y=vor[:, 1], z=vor[:, 2], t=buoy + glat * qc, d=buoy, h=hum, v=torch.ones_like(vol))
    size = nx * ny * (nz + 3)
    acc = {k: torch.zeros(size, dtype=torch.float64, device="cuda") for k in vals}
    for p in _support_points(pos, B, vol):
        u = [(p[:, k] - lower[k]) * dxi[k] for k in range(3)]
        c = [torch.floor(a) for a in u]
        f = [a - b for a, b in zip(u, c)]
        c = [a.long() for a in c]
        for i in range(2):
            for j in range(2):
                for k in range(2):
                    g = (((c[0] + i) % nx) * ny + (c[1] + j) % ny) * (nz + 3) + c[2] + k + 1
                    w = 0.25 * vol
                    for a, m in zip(f, (i, j, k)):
                        w = w * (a if m else 1 - a)
                    for name, v in vals.items():
                        acc[name].index_add_(0, g, w * v)
    acc = {k: a.view(nx, ny, nz + 3) for k, a in acc.items()}
    for a in acc.values():   # free slip: the halo rows fold into the domain
        a[:, :, 1] *= 2
        a[:, :, nz + 1] *= 2
        a[:, :, 2] += a[:, :, 0]
        a[:, :, nz] += a[:, :, nz + 2]
    for name in "xyztdh":
        acc[name][:, :, 1:nz + 2] /= acc["v"][:, :, 1:nz + 2]
    for name in "xyzt":      # linear extrapolation into the halo rows
        a = acc[name]
        a[:, :, 0] = 2 * a[:, :, 1] - a[:, :, 2]
        a[:, :, nz + 2] = 2 * a[:, :, nz + 1] - a[:, :, nz]
    out = {abi.FIELD_NAMES[f]: acc[k] for f, k in zip(P2G_FIELDS, "xyztdhv")}
    c = [torch.floor((pos[:, k] - lower[k]) * dxi[k]).long() for k in range(3)]
    g = (c[0] * ny + c[1]) * (nz + 3) + c[2] + 1
    one = torch.ones_like(vol)
    little = (vol <= 1.0 / (dxi[0] * dxi[1] * dxi[2]) / opts["min_vratio"]).double()
    for f, v in ((abi.NPARG, one), (abi.NSPARG, little)):
        a = torch.zeros(size, dtype=torch.float64, device="cuda")
        out[abi.FIELD_NAMES[f]] = a.index_add_(0, g, v).view(nx, ny, nz + 3)
    return out
