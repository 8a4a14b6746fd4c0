"""The work that users of this package have it do, as measured cases.

Every case is a channel that is advanced through the public entry points
(Lattice, Batch, the C ABI) by the number of steps between two looks at the
fields, and then read: the moments and, with the turbulence model, k and omega,
into the caller's page-locked buffers (as an application that monitors or
writes its run does).  `exact` repeats the same steps in 64 bits with plain
torch: collide, streaming with half-way and interpolated bounce-back, the
k-omega rows, the restarted simpler GMRES at its tolerances, the thermal rows
and BiCGStab, and for the gradient torch's own differentiation.

Kinds:
  step     one lattice, `steps` time steps, fields read
  adjoint  forward of `steps` steps and the gradient of the objective
  batch    several lattices advanced together, fields of all read
"""
import ctypes as C
import math

import numpy as np
import torch

from komegafoulingmodel_b200 import Lattice, _abi, desc_default, shear
from komegafoulingmodel_b200 import geometry as G
from komegafoulingmodel_b200.batch import Batch

STORAGE = {"fp32": _abi.STORE_FP32, "fp64": _abi.STORE_FP64, "fp16row": _abi.STORE_FP16_ROW,
           "fp16neq": _abi.STORE_FP16_NEQ}
NU = {True: 5.0e-4, False: 0.02}  # viscosity with and without the turbulence model


def _case(name, nx, ny, steps, kind="step", komega=True, wave=0.0, storage="fp32", thermal=False):
    return {"name": name, "kind": kind, "nx": nx, "ny": ny, "steps": steps, "komega": komega,
            "wave": wave, "storage": storage, "thermal": thermal}


def listed():
    return [
        # the smallest channel, laminar start-up: launch latency per step
        _case("laminar_256x64", 256, 64, 200, komega=False),
        # an odd-sized laminar channel with curved walls (interpolated bounce-back)
        _case("laminar_wavy_1999x501", 1999, 501, 40, komega=False, wave=24.0),
        # the smallest turbulent channel
        _case("komega_256x64", 256, 64, 20),
        # an ordinary turbulent channel of odd size (one member of a design sweep)
        _case("komega_1001x253", 1001, 253, 20),
        # the turbulent channel with wavy walls
        _case("komega_wavy_2048x256", 2048, 256, 6, wave=32.0),
        # a medium channel, larger than the L2 cache's share of its fields
        _case("komega_4096x512", 4096, 512, 20),
        # the largest: the channel of the headline benchmark
        _case("komega_16384x1024", 16384, 1024, 40),
        # populations stored in 16 bits
        _case("komega_fp16row_8192x512", 8192, 512, 20, storage="fp16row"),
        # everything in 64 bits (precision studies)
        _case("komega_fp64_2048x384", 2048, 384, 10, storage="fp64"),
        # turbulence and temperature together, wavy walls
        _case("thermal_wavy_1536x256", 1536, 256, 6, wave=24.0, thermal=True),
        # wall-shape gradient of a laminar channel: forward and backward
        _case("adjoint_1024x256", 1024, 256, 200, kind="adjoint", komega=False, wave=20.0),
        # channels of uneven size and Reynolds number advanced together
        _case("batch_8", 2048, 256, 6, kind="batch", storage="fp16neq"),
    ]


def draw(rng):
    """A case of the ranges that the listed ones stand for."""
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["laminar", "laminar", "komega", "komega", "komega", "komega", "komega", "fp16row",
                       "fp64", "thermal", "adjoint", "batch"])
    nx, ny = size(200, 16384), size(48, 1024)
    if kind in ("adjoint", "batch", "thermal", "fp64"):
        nx, ny = size(200, 4096), size(48, 384)
    nodes = nx * ny
    most = 0.1 if kind in ("laminar", "adjoint") else 0.05
    wave = rng.choice([0.0, round(rng.uniform(0.02, most) * ny, 2)])
    c = _case("", nx, ny, 0, wave=wave, komega=kind not in ("laminar", "adjoint"),
              storage={"fp16row": "fp16row", "fp64": "fp64", "batch": "fp16neq"}.get(kind, "fp32"),
              thermal=kind == "thermal", kind=kind if kind in ("adjoint", "batch") else "step")
    del c["name"]
    if kind == "laminar":
        c["steps"] = max(10, min(400, int(4.0e7 / nodes)))
    elif kind == "adjoint":
        c["steps"] = rng.randint(60, 200)
        c["wave"] = wave or 0.08 * ny
    elif kind == "batch":
        c["steps"] = 2 * rng.randint(2, 5)
    else:
        c["steps"] = max(6, min(20, int(1.6e8 / nodes)))
        if wave or kind == "thermal":
            c["steps"] = 6
        if kind == "fp16row":
            c["wave"] = 0.0
    return c


# ---- inputs ------------------------------------------------------------------


def _members(case):
    """The lattices of a case (one, or the uneven ones of a batch)."""
    if case["kind"] != "batch":
        return [dict(case, re=1.0)]
    out = []
    for i, (sx, sy, re, ko) in enumerate([(1, 1, 1, True), (0.5, 1, 0.4, True), (0.25, 0.5, 0.2, True),
                                          (1, 0.5, 1, False), (0.5, 0.5, 0.6, True), (0.25, 1, 0.3, False),
                                          (0.75, 0.75, 0.8, True), (0.5, 0.25, 0.5, True)]):
        nx, ny = max(64, int(case["nx"] * sx)), max(34, int(case["ny"] * sy))
        out.append(dict(case, nx=nx, ny=ny, komega=ko, wave=0.0 if ko else 0.06 * ny, re=re))
    return out


def _smooth(gen, ny, nx):
    """A smooth random field in [-1, 1], periodic in x."""
    x = torch.arange(nx, device="cuda", dtype=torch.float64)[None, :] * (2 * math.pi / nx)
    y = torch.arange(ny, device="cuda", dtype=torch.float64)[:, None] * (math.pi / ny)
    a = torch.rand(4, 3, generator=gen, dtype=torch.float64)
    out = torch.zeros(ny, nx, device="cuda", dtype=torch.float64)
    for m in range(4):
        out += (0.5 * float(a[m, 0]) * torch.cos((m + 1) * x + 6.3 * float(a[m, 1]))
                * torch.sin((m + 1) * y + 6.3 * float(a[m, 2])))
    return out


def _phi(c, u):
    return 2.0 / 3.0 - u * u if c == 0 else 0.5 * (1.0 / 3.0 + c * u + u * u)


CX, CY, REV = G.CX.tolist(), G.CY.tolist(), G.REV.tolist()


def _feq(rho, ux, uy):
    px, py = ([_phi(c, u) for c in (0, 1, -1)] for u in (ux, uy))
    return torch.stack([rho * px[CX[q]] * py[CY[q]] for q in range(9)])


def _inputs(m, seed):
    """Walls, parameters and the start state of one lattice, from the seed."""
    nx, ny = m["nx"], m["ny"]
    gen = torch.Generator().manual_seed(seed * 7919 + nx * 31 + ny)
    r = torch.rand(8, generator=gen, dtype=torch.float64).tolist()
    x = np.arange(nx)
    h = np.zeros(nx)
    if m["wave"]:
        periods = max(1, round(nx / 512))
        # a gradient has one value per wall link: its walls are the case's, not the seed's
        amp = m["wave"] * (0.85 + 0.15 * (r[0] if m["kind"] != "adjoint" else 0.5))
        h = 0.5 * amp * (1.0 - np.cos(2 * np.pi * periods * x / nx))
        if m["kind"] == "adjoint":
            h = h + 0.05 * (1.0 - np.cos(2 * np.pi * x / nx)) + 0.1
    yb, yt = 0.5 + h, ny - 1.5 - h
    nu = NU[m["komega"]] / m["re"]
    umax = 0.05 * (0.9 + 0.2 * r[2])
    R = 0.5 * (yt.mean() - yb.mean())
    p = {"nx": nx, "ny": ny, "yb": yb, "yt": yt, "nu": nu, "tau": 1.0 / (3.0 * nu + 0.5),
         "fterm": G.force_from_re((2.0 / 3.0) * umax * R / nu, nu, R), "wave": bool(m["wave"])}
    dev = dict(device="cuda", dtype=torch.float64)
    b, t = torch.tensor(yb, **dev)[None, :], torch.tensor(yt, **dev)[None, :]
    y = torch.arange(ny, **dev)[:, None]
    fluid = (y > b) & (y < t)
    fluid[0] = fluid[-1] = False
    shape = (4.0 * (y - b) * (t - y) / (t - b) ** 2).clamp(min=0.0)
    ux = umax * shape * (1.0 + 0.03 * _smooth(gen, ny, nx))
    uy = 0.02 * umax * shape * _smooth(gen, ny, nx)
    rho = 1.0 + 1.0e-4 * _smooth(gen, ny, nx)
    p["f"] = _feq(rho, ux, uy) * fluid
    zero = torch.zeros_like(ux)
    d = torch.where(fluid, torch.minimum(y - b, t - y), torch.ones_like(ux))
    if m["komega"]:
        # the near-wall behaviour of a running channel: omega ~ 6 nu / (0.075 d^2), k ~ d^2
        k0 = 1.5 * (0.05 * umax) ** 2
        o0 = math.sqrt(k0) / (0.09 ** 0.25 * 0.07 * 2 * R)
        k = k0 * (1.0 - torch.exp(-(d / (0.05 * R + 1.0)) ** 2)) * (1.0 + 0.1 * _smooth(gen, ny, nx))
        o = torch.sqrt(o0 ** 2 + (6.0 * nu / (0.075 * d * d)) ** 2) * (1.0 + 0.05 * _smooth(gen, ny, nx))
        p["k"], p["omega"] = torch.where(fluid, k, zero), torch.where(fluid, o, zero)
        p["nut"] = torch.where(fluid, p["k"] / o, zero)
        sxy = torch.where(fluid, 0.5 * umax * 4.0 * (t + b - 2.0 * y) / (t - b) ** 2, zero)
        p["S"] = torch.stack([zero, sxy, zero])
    if m["thermal"]:
        x = torch.arange(nx, **dev)[None, :] / nx
        p["T"] = torch.where(fluid, 2.0 * (1.0 - torch.exp(-d / (0.2 * R))) * (1.0 - 0.3 * x), zero)
    return p


def _host(t):
    return t.cpu().numpy().reshape(-1)


def _open(m, p):
    """A lattice with the case's walls and start state loaded."""
    d = desc_default()
    d.nx, d.nx_full, d.ny = p["nx"], p["nx"], p["ny"]
    d.tau, d.fterm, d.mu = p["tau"], p["fterm"], p["nu"]
    d.use_komega, d.use_thermal = int(m["komega"]), int(m["thermal"])
    d.storage = STORAGE[m["storage"]]
    L = Lattice(d)
    torch.cuda.synchronize()
    if m["storage"] == "fp64":  # takes its geometry from the host builder
        ch = G.channel_from_walls(p["nx"], p["ny"], p["yb"], p["yt"], wall_distance=not p["wave"])
        if p["wave"]:
            ch.wallD = _geometry(p)["wallD"].cpu().numpy().reshape(-1)
        L.set_geometry(ch.ntype, ch.wallD, ch.dX, ch.ibb_idx if len(ch.ibb_idx) else None,
                       ch.ibb_q if len(ch.ibb_q) else None)
    else:
        L.set_walls(p["yb"], p["yt"], ibb_all=m["kind"] == "adjoint")
    if m["komega"]:
        L.set_state(*(_host(p[k]) for k in ("f", "k", "omega", "nut", "S")))
    else:
        L.set_state(_host(p["f"]))
    if m["thermal"]:
        L.set_temperature(_host(p["T"]))
    return L


def _shear_setup(p):
    ch = G.channel_from_walls(p["nx"], p["ny"], p["yb"], p["yt"], ibb_all=True, wall_distance=False)
    nodes, col = shear.shear_nodes(ch)
    return shear.ShearSetup(nodes, col, shear.shear_coeffs(ch, nodes), np.zeros((0, 4), np.int32), np.zeros((0, 4)))


def prepare(case, seed):
    ms = _members(case)
    lats, bufs = [], []
    for i, m in enumerate(ms):
        p = _inputs(m, seed + 1000 * i)
        L = _open(m, p)
        if case["kind"] == "adjoint":
            L.set_shear(_shear_setup(p))
        if case["kind"] != "step":
            L.step(1)
            L.sync()
        planes = 9 if case["kind"] == "adjoint" else 3 + 2 * m["komega"] + m["thermal"]
        bufs.append(torch.zeros(planes, m["ny"], m["nx"], dtype=torch.float64, pin_memory=True))
        lats.append(L)
    return {"case": dict(case), "members": ms, "lattices": lats, "buffers": bufs,
            "batch": Batch(lats) if case["kind"] == "batch" else None}


# ---- one pass ----------------------------------------------------------------


def _ptr(t):
    return C.cast(t.data_ptr(), C.POINTER(C.c_double))


def _read(m, L, buf):
    """The fields into the caller's page-locked buffer: density, velocity,
    and k, omega and the temperature where the lattice has them."""
    _abi.check("kofm_get_macro", L.lib.kofm_get_macro(L._ctx, _ptr(buf[0]), _ptr(buf[1]), _ptr(buf[2])))
    out = {"rho": buf[0], "u": buf[1:3]}
    if m["komega"]:
        _abi.check("kofm_get_state", L.lib.kofm_get_state(L._ctx, None, _ptr(buf[3]), _ptr(buf[4]), None, None))
        out["k"], out["omega"] = buf[3], buf[4]
    if m["thermal"]:
        _abi.check("kofm_get_temperature", L.lib.kofm_get_temperature(L._ctx, _ptr(buf[5])))
        out["T"] = buf[5]
    return out


def run(state):
    case, lats = state["case"], state["lattices"]
    if case["kind"] == "adjoint":
        J, dq = lats[0].adjoint(case["steps"])
        f = state["buffers"][0]
        _abi.check("kofm_get_state", lats[0].lib.kofm_get_state(lats[0]._ctx, _ptr(f), None, None, None, None))
        return {"J": J, "dJdq": dq, "f": f}
    if case["kind"] == "batch":
        state["batch"].step(case["steps"])
    else:
        lats[0].step(case["steps"])
    return [_read(m, L, b) for m, L, b in zip(state["members"], lats, state["buffers"])]


def work(case):
    """Per node and step the state read once and written once: populations,
    flags and moments; with the turbulence model k, omega, the strain rates,
    the wall distance and nu_t; the adjoint reads and writes the adjoint
    populations beside the stored states.  The fields of the read-out once."""
    total = flops = 0.0
    for m in _members(case):
        pop = {"fp32": 4, "fp64": 8}.get(m["storage"], 2)
        fld = 8 if m["storage"] == "fp64" else 4
        b = 18.0 * pop + 2.0 + 3.0 * fld
        fl = 250.0
        if m["komega"]:
            b += fld * (2 * 2 + 2 * 3 + 1 + 1)
            fl += 900.0
        if m["thermal"]:
            b += 16.0
            fl += 200.0
        if case["kind"] == "adjoint":
            b, fl = 36.0 * 5, 900.0
        nodes = m["nx"] * m["ny"]
        read = 9 if case["kind"] == "adjoint" else 3 + 2 * m["komega"] + m["thermal"]
        total += nodes * (b * m["steps"] + 8.0 * read)
        flops += nodes * fl * m["steps"]
    return {"bytes": total, "flops": flops}


def tolerance(case):
    """Largest differences between two correct implementations, about four
    times those measured between the solver's forms and against 64 bits: the
    rounding of the stored fields, and with the turbulence model the GMRES
    cycles' cuts (relative tolerance 1e-4), which move with the order of a sum;
    curved walls amplify both."""
    if case["storage"] in ("fp16row", "fp16neq"):
        return {"rel": 1.0e-3 if case["wave"] or case["kind"] == "batch" else 1.0e-4}
    if not case["komega"]:
        return {"rel": 1.0e-6}
    return {"rel": 2.0e-4 if case["wave"] else 5.0e-6}


# ---- the same in 64 bits with plain torch --------------------------------------


def _nb(a, q):
    """The field at the neighbour in direction q (rows 0 and ny-1 are walls)."""
    return torch.roll(a, shifts=(-CY[q], -CX[q]), dims=(-2, -1))


def _geometry(p, keep_half=False):
    nx, ny = p["nx"], p["ny"]
    dev = dict(device="cuda", dtype=torch.float64)
    walls = [torch.tensor(p[k], **dev) for k in ("yb", "yt")]
    y = torch.arange(ny, **dev)[:, None]
    fluid = (y > walls[0]) & (y < walls[1])
    fluid[0] = fluid[-1] = False
    g = {"fluid": fluid, "wall": [None], "frac": [None], "ibb": [None]}
    seam = torch.zeros(nx, dtype=torch.bool, device="cuda")
    seam[0] = seam[-1] = True
    for q in range(1, 9):
        hit = fluid & ~_nb(fluid, q)
        best = torch.full((ny, nx), math.inf, **dev)
        for w in walls:
            d = torch.roll(w, -CX[q]) - w if CX[q] else torch.zeros_like(w)
            t = (w - y) / (CY[q] - d)
            best = torch.where((t > 0) & (t <= 1 + 1e-12), torch.minimum(best, t.clamp(max=1.0)), best)
        frac = torch.where(torch.isfinite(best), best, 0.5)
        g["wall"].append(hit)
        g["frac"].append(frac)
        g["ibb"].append(hit & ~seam & (keep_half | ((frac - 0.5).abs() > 1e-12)))
    one = torch.ones(ny, nx, **dev)
    g["dX"] = [torch.where(g["wall"][q], g["frac"][q].clamp(min=0.001), one) for q in range(1, 5)]
    g["wallD"] = _wall_distance(p, walls, y, fluid)
    return g


def _wall_distance(p, walls, y, fluid, radius=50):
    """Distance to the wall segments within `radius` columns: to a segment's
    line, or to an end where the foot of the perpendicular on the segment's
    normal side falls beyond that end in x."""
    nx = p["nx"]
    if not p["wave"]:
        return torch.where(fluid, torch.minimum(y - walls[0], walls[1] - y), torch.zeros_like(y))
    i = torch.arange(nx, device="cuda")
    x = i.double()
    best = torch.full(fluid.shape, 1000.0, device="cuda", dtype=torch.float64)
    for top in (False, True):
        w = walls[int(top)]
        lo, hi = (-radius + 1, radius) if top else (-radius, radius - 1)
        for o in range(lo, hi + 1):
            xa = i + o
            there = (xa >= -1) & (xa <= nx - 1)
            ax, ay, by = xa.double(), w[xa % nx], w[(xa + 1) % nx]
            P0, P1 = ((ax + 1, by), (ax, ay)) if top else ((ax, ay), (ax + 1, by))
            tx, ty = P1[0] - P0[0], P1[1] - P0[1]
            mag = torch.sqrt(tx * tx + ty * ty)
            d = (ty * x - tx * y + P1[0] * P0[1] - P1[1] * P0[0]).abs() / mag
            foot = x + d * (ty / mag)
            c0 = foot > P0[0] if top else foot < P0[0]
            c1 = ~c0 & (foot < P1[0] if top else foot > P1[0])
            d = torch.where(c0, torch.hypot(x - P0[0], y - P0[1]), d)
            d = torch.where(c1, torch.hypot(x - P1[0], y - P1[1]), d)
            best = torch.where(there & (d < best), d, best)
    return torch.where(fluid, best, torch.zeros_like(best))


def _moments(f, fluid):
    rho = torch.where(fluid, f.sum(0), torch.ones((), device="cuda", dtype=torch.float64))
    ux = (f[1] - f[2] + f[5] - f[6] + f[7] - f[8]) / rho
    uy = (f[3] - f[4] + f[5] - f[6] - f[7] + f[8]) / rho
    return rho, ux, uy


def _stream(fs, g, frac=None):
    """Post-stream populations: half-way bounce-back, then Bouzidi's linear
    interpolation on the listed links."""
    frac = frac or g["frac"]
    new = [fs[0]]
    for q in range(1, 9):
        new.append(torch.where(g["wall"][REV[q]], fs[REV[q]], _nb(fs[q], REV[q])))
    out = list(new)
    for q in range(1, 9):
        q2, r = 2.0 * frac[q], REV[q]
        near = q2 * new[r] + (1.0 - q2) * new[q]
        far = (new[r] + (q2 - 1.0) * fs[r]) / q2
        out[r] = torch.where(g["ibb"][q], torch.where(q2 <= 1.0, near, far), new[r])
    return torch.stack(out)


def _weights(a, b):
    a, b = a.clamp(min=0.1), b.clamp(min=0.1)
    s = a + b
    c = (a - b) / (a * b)
    far = c.abs() > 10.0
    d1 = [torch.where(far, 1.0 / s, b / (a * s)), torch.where(far, -1.0 / s, -a / (b * s)),
          torch.where(far, torch.zeros_like(c), c)]
    return d1, [2.0 / (a * s), 2.0 / (b * s), -2.0 / (a * b)]


class _Exact:
    """One lattice in 64 bits."""

    SST = dict(bs=0.09, k1=0.85, k2=1.0, o1=0.5, o2=0.856, a1=0.31, kappa=0.41, c=0.5477225575,
               g1=5.0 / 9.0, g2=0.44)

    def __init__(self, m, p, keep_half=False):
        self.m, self.p, self.g = m, p, _geometry(p, keep_half)
        self.fluid = self.g["fluid"]
        self.f = p["f"]
        if m["komega"]:
            self.k, self.o = p["k"].clone(), p["omega"].clone()
            self.S = list(p["S"])
            self.X, self.X2 = _weights(self.g["dX"][0], self.g["dX"][1])
            self.Y, self.Y2 = _weights(self.g["dX"][2], self.g["dX"][3])
            self.near = (self.g["wall"][1] | self.g["wall"][2] | self.g["wall"][3] | self.g["wall"][4])
        if m["thermal"]:
            self.T = p["T"].clone()

    def on(self, a):
        return torch.where(self.fluid, a, torch.zeros_like(a))

    def collide(self, f):
        p, fl, m = self.p, self.fluid, self.SST
        rho, ux, uy = _moments(f, fl)
        w = p["tau"]
        if self.m["komega"]:
            self.o = self.o.abs()
            self.k = torch.where(self.k < 0, torch.full_like(self.k, 1e-16), self.k)
            yw = torch.where(fl, self.g["wallD"], torch.ones_like(rho))
            o = torch.where(fl, self.o, torch.ones_like(rho))
            a = torch.maximum(2.0 * self.k.sqrt() / (m["bs"] * o * yw), 500.0 * p["nu"] / (yw * yw * o))
            S = self.S
            F2 = torch.tanh(a * a) * torch.sqrt(2.0 * (S[0] ** 2 + 2.0 * S[1] ** 2 + S[2] ** 2))
            nut = (m["a1"] * self.k / torch.maximum(m["a1"] * o, F2)).clamp(max=10.0).clamp(min=1e-16)
            self.nut = self.on(nut)
            w = 1.0 / (3.0 * (nut + p["nu"]) + 0.5)
        feq = _feq(rho, ux, uy)
        neq = f - feq
        self.rho, self.ux, self.uy = self.on(rho), self.on(ux + 0.5 * p["fterm"]), self.on(uy)
        if self.m["komega"]:
            s = -1.5 * p["tau"] / rho
            self.S = [self.on(s * sum(wt[q] * neq[q] for q in range(9) if wt[q])) for wt in
                      ([c * c for c in CX], [a * b for a, b in zip(CX, CY)], [c * c for c in CY])]
        return (f - w * neq - feq + _feq(rho, ux + p["fterm"], uy)) * fl

    def rows(self):
        """The normalised backward-Euler rows of omega and k and b - A x."""
        m, fl, X, Y, X2, Y2 = self.SST, self.fluid, self.X, self.Y, self.X2, self.Y2
        mu, one = self.p["nu"], torch.ones_like(self.k)
        k, o, nut, rho = self.k, self.o, self.nut, torch.where(fl, self.rho, one)
        oc, yw = torch.where(fl, o, one), torch.where(fl, self.g["wallD"], one)

        def grad(a):
            return (X[0] * _nb(a, 1) + X[1] * _nb(a, 2) + X[2] * a, Y[0] * _nb(a, 3) + Y[1] * _nb(a, 4) + Y[2] * a)

        do, dk = grad(o), grad(k)
        cross = [2.0 * m["o2"] / oc * d for d in dk]
        cd = (rho * (cross[0] * do[0] + cross[1] * do[1])).clamp(min=1e-10)
        a = torch.maximum(k.clamp(min=0).sqrt() / (m["bs"] * oc * yw), 500.0 * mu / (yw * yw * oc))
        a = torch.minimum(a, 4.0 * k * m["o2"] / (cd * yw * yw))
        F1 = torch.tanh(a ** 4)
        Dk = self.on(mu + (m["k1"] * F1 + m["k2"] * (1 - F1)) * nut)
        Do = self.on(mu + (m["o1"] * F1 + m["o2"] * (1 - F1)) * nut)
        gk, go = grad(Dk), grad(Do)
        S = self.S
        kv, om = k.clamp(min=0), o.clamp(min=0)
        Pk = 2.0 * nut * (S[0] ** 2 + S[2] ** 2 + 2.0 * S[1] ** 2) - 2.0 / 3.0 * kv * rho * (S[0] + S[2])
        Pk = torch.minimum(Pk, 10.0 * m["bs"] * kv * om).clamp(min=0)
        gam = (F1 * m["g1"] + (1 - F1) * m["g2"]) / torch.where(fl, nut, one)
        sink = m["bs"] * om
        wall_o = torch.sqrt((6.0 * mu / 0.075 / (yw * yw)) ** 2 + (kv.sqrt() / (m["c"] * m["kappa"] * yw)) ** 2)
        dt = torch.where(self.near, 0.0, 1.0).double()
        zero = torch.zeros_like(k)
        out = []
        for D, J, step, snk, src, x in (
                (Do, (self.ux - go[0] - cross[0], self.uy - go[1] - cross[1]), dt,
                 torch.where(self.near, zero, sink),
                 torch.where(self.near, wall_o.clamp(max=1000.0), om + gam * Pk), o),
                (Dk, (self.ux - gk[0], self.uy - gk[1]), one, sink, kv + Pk, k)):
            diag = 1.0 + step * (J[0] * X[2] + J[1] * Y[2] - D * (X2[2] + Y2[2])) + snk
            A = [self.on(step * c / diag) for c in (J[0] * X[0] - D * X2[0], J[0] * X[1] - D * X2[1],
                                                    J[1] * Y[0] - D * Y2[0], J[1] * Y[1] - D * Y2[1])]
            out.append((A, self.on(src / diag) - self.matvec(A, x)))
        return out

    @staticmethod
    def matvec(A, x):
        return A[3] * _nb(x, 4) + A[1] * _nb(x, 2) + x + A[0] * _nb(x, 1) + A[2] * _nb(x, 3)

    def gmres(self, A, b, K=10, rel=1e-4, atol=1e-7):
        """Restarted simpler GMRES (Walker & Zhou): each cycle ends at the first
        vector that the tests on diag(R) or on xi refuse."""
        def dot(u, v):
            return float(torch.dot(u.reshape(-1), v.reshape(-1)))

        x, norm = torch.zeros_like(b), math.sqrt(dot(b, b))
        for restart in range(100):
            r = b - self.matvec(A, x) if restart else b
            rho0 = math.sqrt(dot(r, r))
            if norm == 0.0 or rho0 / norm <= rel or rho0 <= atol:
                break
            r = r / rho0
            V, xi, R, rho, k = [], [], [0.0] * (K * K), 1.0, K
            full = K
            for i in range(K):
                v = self.matvec(A, V[-1] if V else r)
                h = [dot(v, u) for u in V]
                for c, u in zip(h, V):
                    v = v - c * u
                n = math.sqrt(dot(v, v))
                for j, c in enumerate(h):
                    R[j + i * K] = c
                R[i + i * K] = n
                V.append(v / n if n else v)
                xi.append(dot(r, V[-1]))
                if n < rel * R[0]:
                    k = full = i
                    break
                if abs(xi[i]) >= rho:
                    k = i
                    break
                rho *= math.sin(math.acos(xi[i] / rho))
            for i in range(k - 1, -1, -1):
                for j in range(i + 1, k):
                    xi[i] -= R[i + j * full] * xi[j]
                xi[i] /= R[i + i * full]
            c = [v * rho0 for v in xi[:k]] + xi[k:]
            x = x + c[0] * r
            for j in range(1, k):
                x = x + c[j] * V[j - 1]
        return x

    def thermal(self):
        """Backward-Euler rows of the temperature (inlet x = 0, outlet
        x = nx - 1) and the reference's BiCGStab with omega = 1."""
        p, fl, dX = self.p, self.fluid, self.g["dX"]
        X, X2 = _weights(dX[0], dX[1])
        Y, Y2 = _weights(dX[2], dX[3])
        prt, nut = 1.0 / 0.9, self.nut
        at = nut * prt
        Jx = self.ux - prt * (X[0] * _nb(nut, 1) + X[1] * _nb(nut, 2) + X[2] * at)
        Jy = self.uy - prt * (Y[0] * _nb(nut, 3) + Y[1] * _nb(nut, 4) + Y[2] * at)
        al = p["nu"] / 0.708 + at
        src = self.T.clamp(min=0.0).clamp(max=2.0)
        diag = 1.0 + Jx * X[2] + Jy * Y[2] - al * (X2[2] + Y2[2])
        A = [Jx * X[0] - al * X2[0], Jx * X[1] - al * X2[1], Jy * Y[0] - al * Y2[0], Jy * Y[1] - al * Y2[1]]
        src[:, 0] -= 2.0 * A[1][:, 0]
        diag[:, -1] += A[0][:, -1]
        A = [self.on(a / diag) for a in A]
        A[1][:, 0] = 0.0
        A[0][:, -1] = 0.0
        b, x = self.on(src / diag), self.T
        nb = float(b.abs().sum())
        b = b - self.matvec(A, x)
        r0, pv, first = b, b, None
        rho = float((b * b).sum())
        for it in range(1000):
            if it:
                new = float((b * r0).sum())
                pv = b + (new / rho) * alpha * (pv - v)
                rho = new
            v = self.matvec(A, pv)
            alpha = rho / float((v * r0).sum())
            x, b = x + alpha * pv, b - alpha * v
            res = float(b.abs().sum()) / nb
            first = res if first is None else first
            if res <= 1e-4 or res <= 1e-7 * first:
                break
            x, b = x + b, b - self.matvec(A, b)
            res = float(b.abs().sum()) / nb
            if res <= 1e-4 or res <= 1e-7 * first:
                break
        self.T = x

    def step(self):
        self.f = _stream(self.collide(self.f), self.g)
        if self.m["komega"]:
            sol = [self.gmres(A, b) for A, b in self.rows()]
            self.o, self.k = self.on(self.o + sol[0]), self.on(self.k + sol[1])
        if self.m["thermal"]:
            self.thermal()

    def out(self):
        o = {"rho": self.rho, "u": torch.stack([self.ux, self.uy])}
        if self.m["komega"]:
            o["k"], o["omega"] = self.k, self.o
        if self.m["thermal"]:
            o["T"] = self.T
        return o


def _exact_adjoint(m, p):
    """J and dJ/dq of the listed links by torch's differentiation, one step of
    the forward recomputed at a time."""
    from torch.utils.checkpoint import checkpoint
    sim = _Exact(m, p, keep_half=True)
    g, fl = sim.g, sim.fluid
    sh = _shear_setup(p)
    nodes = torch.tensor(np.asarray(sh.nodes), device="cuda", dtype=torch.int64)
    rows = torch.tensor(sh.cfss, device="cuda", dtype=torch.float64).reshape(-1, 2, 8)
    frac = [None] + [g["frac"][q].clone().requires_grad_(True) for q in range(1, 9)]
    visc = p["nu"] / (3.0 * p["nu"] + 0.5)
    ends = [fl[:, 0].double(), fl[:, -1].double()]

    def one(fs, *fr):
        f = _stream(fs, g, [None, *fr])
        rho, ux, uy = _moments(f, fl)
        j = ((rho[:, 0] * ends[0]).sum() / ends[0].sum() - (rho[:, -1] * ends[1]).sum() / ends[1].sum()) / 3.0
        r, u, v = (a.reshape(-1)[nodes] for a in (rho, ux, uy))
        neq = f.reshape(9, -1)[:, nodes] - _feq(r, u + 0.5 * p["fterm"], v)
        tx = (neq[1:] * rows[:, 0].T).sum(0)
        ty = (neq[1:] * rows[:, 1].T).sum(0)
        tau = torch.sqrt(tx * tx + ty * ty) * visc / r
        j = j + torch.where(tx < 0, -tau, tau).sum()
        feq = _feq(rho, ux, uy)
        return (f - p["tau"] * (f - feq) - feq + _feq(rho, ux + p["fterm"], uy)) * fl, j

    fs, J = sim.collide(p["f"]), 0.0
    for _ in range(m["steps"]):
        fs, j = checkpoint(one, fs, *frac[1:], use_reentrant=False)
        J = J + j
    J.backward()
    dq = torch.cat([frac[q].grad[g["ibb"][q]] for q in range(1, 9)])
    with torch.no_grad():
        f = sim.on(_stream(fs, g))
    return {"J": float(J.detach()), "dJdq": dq.cpu().numpy(), "f": f}


def exact(case, seed):
    outs = []
    for i, m in enumerate(_members(case)):
        p = _inputs(m, seed + 1000 * i)
        if case["kind"] == "adjoint":
            return _exact_adjoint(m, p)
        sim = _Exact(m, p)
        with torch.no_grad():
            for _ in range(case["steps"] + (case["kind"] == "batch")):
                sim.step()
            outs.append({k: v.cpu() for k, v in sim.out().items()})
    return outs
