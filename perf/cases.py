"""What is measured of the engine: projections, time steps, transport and serving as a user's program calls them.

Sizes and settings are those of the benchmark configurations (synth.py) and of the tests, with odd
and ragged ones among them; inputs are drawn from a seed on the GPU. ``exact`` restates each
path in 64-bit torch from the case alone (geometry, face kinds, operator, momentum, transport).
"""
import json
import math
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import torch

import __graft_entry__ as entry

pkg = entry.package()

DEV = torch.device("cuda" if torch.cuda.is_available() else "cpu")
F64 = torch.float64
INTERIOR, WALL, SLIP, INLET, OUTLET, BLOCKED = range(6)
TOL = 1e-8  # every benchmark configuration solves to this relative residual
MAX_ITER = 10000


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # The smallest call: one parity-form projection of a coarse trial grid with one building.
        {"name": "project-ic0-24x20x16", "kind": "project", "form": "ic0", "cells": "24x20x16", "dx": 1.0, "inflow": 1.0,
         "boxes": 1, "dt": 1.0},
        # The first configuration: a uniform 64x64x32 grid without buildings, IC(0) to 1e-8.
        {"name": "project-ic0-64x64x32", "kind": "project", "form": "ic0", "cells": "64x64x32", "dx": 1.0, "inflow": 1.0,
         "boxes": 0, "dt": 1.0},
        # The second configuration's projection in the parity form: 12 buildings, multigrid.
        {"name": "project-multigrid-128x128x64", "kind": "project", "form": "multigrid", "cells": "128x128x64", "dx": 2.0,
         "inflow": 5.0, "boxes": 12, "dt": 0.1},
        # A laminar time step in the parity form on an odd grid whose spacing is no power of two.
        {"name": "step-multigrid-75x61x37", "kind": "step", "form": "multigrid", "cells": "75x61x37", "dx": 1.5,
         "inflow": 5.0, "boxes": 4, "dt": 0.1},
        # One mid-sized case alone in the mixed form, rows no multiple of 16 cells.
        {"name": "project-mixed-100x84x50", "kind": "project", "form": "mixed", "cells": "100x84x50", "dx": 2.0,
         "inflow": 5.0, "boxes": 8, "dt": 0.1},
        # The third configuration: one large mixed-precision solve, 8.4 M cells, 40 buildings.
        {"name": "project-mixed-256x256x128", "kind": "project", "form": "mixed", "cells": "256x256x128", "dx": 2.0,
         "inflow": 5.0, "boxes": 40, "dt": 0.1},
        # The second configuration as it is run in the mixed form: a laminar SSPRK2 time step.
        {"name": "step-mixed-128x128x64", "kind": "step", "form": "mixed", "cells": "128x128x64", "dx": 2.0,
         "inflow": 5.0, "boxes": 12, "dt": 0.1},
        # The fourth configuration: uneven grids with 0-20 buildings in one batched call.
        {"name": "batch-uneven-8", "kind": "batch", "shapes": "48x48x48 64x64x32 96x96x48 128x128x64 160x160x80 64x64x32 96x96x48 128x128x64",
         "dx": 2.0, "inflow": 5.0, "boxes": 20, "dt": 0.1},
        # The fifth configuration: wind directions over one built-up site and smaller cases
        # beside them, served from host buffers through the continuous-batching server.
        {"name": "serve-wind-16", "kind": "serve", "cells": "128x128x64", "directions": 10, "small": "96x96x48", "smalls": 6,
         "dx": 2.0, "boxes": 30, "dt": 0.1},
        # Dispersion on a projected flow: one linear-upwind step of a constituent, receptors read.
        {"name": "scalar-upwind-128x128x64", "kind": "scalar", "muscl": False, "cells": "128x128x64", "dx": 2.0,
         "inflow": 5.0, "boxes": 12, "receptors": 6},
        # The same with MUSCL and the mass budget, on an odd grid with a spacing of 1.5 m.
        {"name": "scalar-muscl-90x70x45", "kind": "scalar", "muscl": True, "cells": "90x70x45", "dx": 1.5,
         "inflow": 5.0, "boxes": 6, "receptors": 6},
        # A thin layered domain whose cells are ten times flatter than wide (line smoothing), to
        # the round-off tolerance of the reference's anisotropic campaign.
        {"name": "solve-anisotropic-48x48x48", "kind": "solve", "cells": "48x48x48", "thin": 0.1},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _cells(rng, lo, hi):
    """Grid sizes spread over their logarithm between the two shapes, odd ones among them."""
    return "x".join(str(_log(rng, lo[a], hi[a])) for a in range(3))


def draw(rng):
    kind = rng.choice(["ic0", "multigrid", "mixed", "step", "batch", "serve", "scalar", "solve"])
    dx, dt = rng.choice([1.0, 1.5, 2.0, 2.5]), rng.choice([0.05, 0.1, 0.25])
    if kind in ("ic0", "multigrid", "mixed"):
        lo, hi = {"ic0": ((16, 16, 8), (96, 96, 48)), "multigrid": ((16, 16, 8), (128, 128, 64)),
                  "mixed": ((32, 32, 16), (200, 200, 100))}[kind]
        return {"kind": "project", "form": kind, "cells": _cells(rng, lo, hi), "dx": dx, "inflow": rng.choice([1.0, 5.0]),
                "boxes": rng.randrange(0, 21), "dt": dt}
    if kind == "step":
        form = rng.choice(["multigrid", "mixed"])
        hi = (80, 80, 40) if form == "multigrid" else (160, 160, 80)
        return {"kind": "step", "form": form, "cells": _cells(rng, (24, 24, 12), hi), "dx": dx,
                "inflow": 5.0, "boxes": rng.randrange(0, 13), "dt": 0.1 if dx >= 2 else 0.05}
    if kind == "batch":
        shapes = [rng.choice(["48x48x48", "64x64x32", "96x96x48", "128x128x64", _cells(rng, (32, 32, 16), (128, 128, 64))])
                  for _ in range(rng.randrange(2, 9))]
        return {"kind": "batch", "shapes": " ".join(shapes), "dx": 2.0, "inflow": 5.0, "boxes": 20, "dt": dt}
    if kind == "serve":
        return {"kind": "serve", "cells": rng.choice(["64x64x32", "96x96x48", "112x100x60"]), "directions": rng.randrange(2, 11),
                "small": rng.choice(["48x48x48", "64x64x32", "72x56x40"]), "smalls": rng.randrange(0, 7), "dx": 2.0,
                "boxes": rng.randrange(5, 31), "dt": dt}
    if kind == "scalar":
        return {"kind": "scalar", "muscl": rng.random() < 0.5, "cells": _cells(rng, (24, 24, 12), (192, 192, 96)), "dx": dx,
                "inflow": 5.0, "boxes": rng.randrange(0, 21), "receptors": rng.randrange(1, 13)}
    return {"kind": "solve", "cells": "x".join(str(_log(rng, 16, h)) for h in (56, 56, 48)),
            "thin": rng.choice([0.05, 0.1, 0.15])}


# ------------------------------------------------------------------ a case's grids
def _shape(text):
    return tuple(int(v) for v in text.split("x"))


def _boxes(seed, count, cells, dx):
    """Ground-based buildings: footprint sides 10-30 m, heights 10-60 m below the domain top."""
    rng = np.random.default_rng(seed)
    lx, ly, lz = (v * dx for v in cells)
    out = []
    for _ in range(count):
        sx, sy = (min(rng.uniform(10.0, 30.0), 0.4 * size) for size in (lx, ly))
        h = max(min(rng.uniform(10.0, 60.0), lz - 2.0 * dx), dx)
        x0, y0 = rng.uniform(0.0, lx - sx), rng.uniform(0.0, ly - sy)
        out.append(((x0, y0, 0.0), (x0 + max(sx, dx), y0 + max(sy, dx), h)))
    return out


def _sites(case):
    """One dict per grid of the case: cells, spacing, boundaries, buildings and flow."""
    open_x = ("open", "wall", "wall")
    k = case["kind"]
    if k == "batch":
        out = []
        for i, s in enumerate(case["shapes"].split()):
            cells, count = _shape(s), (7 * i + 3) % (case["boxes"] + 1)
            out.append({"cells": cells, "dx": case["dx"], "bnd": open_x, "inflow": case["inflow"],
                        "boxes": _boxes(100 + i, count, cells, case["dx"])})
        return out
    if k == "serve":
        cells, small = _shape(case["cells"]), _shape(case["small"])
        boxes = _boxes(4, case["boxes"], cells, case["dx"])
        out = [{"cells": cells, "dx": case["dx"], "bnd": ("open", "open", "ground_open_top"), "inflow": 5.0, "boxes": boxes,
                "direction": 10.0 * (36 * d // case["directions"])} for d in range(case["directions"])]
        for i in range(case["smalls"]):
            out.append({"cells": small, "dx": case["dx"], "bnd": open_x, "inflow": 5.0,
                        "boxes": _boxes(4000 + i, (5 * i) % 21, small, case["dx"])})
        return out
    cells = _shape(case["cells"])
    return [{"cells": cells, "dx": case["dx"], "bnd": open_x, "inflow": case["inflow"],
             "boxes": _boxes(1, case["boxes"], cells, case["dx"])}]


def _framework_case(site, preconditioner):
    c = pkg.synth.case(site["cells"], site["dx"], boundaries=site["bnd"], inflow=site["inflow"], boxes=site["boxes"],
                       preconditioner=preconditioner)
    if "direction" in site:
        c["flow"] = {"kind": "neutral_rans", "speed_m_s": site["inflow"], "reference_height_m": 10.0, "roughness_m": 0.1,
                     "direction_deg_from": site["direction"], "viscosity_m2_s": 1.5e-5, "turbulent_schmidt": 0.7}
    return c


def _thin_case(case):
    c = pkg.synth.case(_shape(case["cells"]), 1.0, boundaries=("wall", "periodic", "wall"), inflow=0.0,
                       preconditioner="multigrid")
    c["domain"]["size_m"] = [1.0, 1.0, case["thin"]]
    return c


class Topo:
    """Solid cells and face kinds of a site, as [z][y][x] tensors."""

    def __init__(self, site):
        nx, ny, nz = self.n = site["cells"]
        self.dx = site["dx"]
        solid = np.zeros((nz, ny, nx), dtype=bool)
        for lo, hi in site["boxes"]:
            cut = []
            for a in range(3):
                centres = (np.arange(self.n[a]) + 0.5) * self.dx
                cut.append(slice(int((centres < lo[a]).sum()), int((centres < hi[a]).sum())))
            solid[cut[2], cut[1], cut[0]] = True
        self.fluid = torch.from_numpy(~solid).to(DEV)
        self.kind, self.vel = [], []
        for a in range(3):
            d = 2 - a
            pad = torch.zeros_like(self.fluid.narrow(d, 0, 1))
            lo, hi = torch.cat([pad, self.fluid], d), torch.cat([self.fluid, pad], d)
            kind = torch.full(lo.shape, BLOCKED, dtype=torch.uint8, device=DEV)
            kind[lo & hi] = INTERIOR
            kind[lo ^ hi] = WALL
            z = torch.arange(lo.shape[0], dtype=F64, device=DEV) + (0.0 if a == 2 else 0.5)
            vel = self._flow(site, z * self.dx)[a].reshape(-1, 1, 1).expand(lo.shape)
            for end, normal in ((0, -1.0), (self.n[a], 1.0)):
                k, live = kind.narrow(d, end, 1), (lo ^ hi).narrow(d, end, 1)
                b = site["bnd"][a]
                if b == "open":
                    v = vel.narrow(d, end, 1) * normal
                    k[live] = SLIP
                    k[live & (v < -1e-12)] = INLET
                    k[live & (v > 1e-12)] = OUTLET
                elif b == "ground_open_top" and end:
                    k[live] = SLIP
            self.kind.append(kind)
            self.vel.append(vel)
        w = 1.0 / self.dx ** 2
        self.w = [(self.kind[a].narrow(2 - a, 1, self.n[a] - 1) == INTERIOR).to(F64) * w for a in range(3)]
        self.diag = torch.zeros(self.fluid.shape, dtype=F64, device=DEV)
        for a in range(3):
            f = (self.kind[a] == INTERIOR).to(F64) * w + (self.kind[a] == OUTLET).to(F64) * 2.0 * w
            self.diag += (f.narrow(2 - a, 0, self.n[a]) + f.narrow(2 - a, 1, self.n[a])) * self.fluid

    @staticmethod
    def _flow(site, z):
        zero = torch.zeros_like(z)
        if "direction" not in site:
            return zero + site["inflow"], zero, zero
        speed = site["inflow"] * torch.log((z.clamp(min=0.0) + 0.1) / 0.1) / math.log((10.0 + 0.1) / 0.1)
        t = site["direction"] * (math.pi / 180.0)
        return -speed * math.sin(t), -speed * math.cos(t), zero

    def faces(self, flat):
        at, out = 0, []
        for k in self.kind:
            out.append(flat[at:at + k.numel()].reshape(k.shape))
            at += k.numel()
        return out

    @staticmethod
    def flat(faces):
        return torch.cat([f.reshape(-1) for f in faces])

    def lohi(self, a, x):
        """The cell values below and above each face of axis a, 0 outside the domain and in solids."""
        d = 2 - a
        x = torch.where(self.fluid, x, 0.0)
        pad = torch.zeros_like(x.narrow(d, 0, 1))
        return torch.cat([pad, x], d), torch.cat([x, pad], d)

    def fixed(self, u):
        """The face values of walls and inlets, in place of u's."""
        out = []
        for f, k, v in zip(u, self.kind, self.vel):
            f = torch.where((k == INTERIOR) | (k == OUTLET), f, 0.0)
            out.append(torch.where(k == INLET, v, f))
        return out

    def apply(self, x):
        y = self.diag * x
        for a in range(3):
            d, m = 2 - a, self.n[a] - 1
            y.narrow(d, 1, m).addcmul_(self.w[a], x.narrow(d, 0, m), value=-1.0)
            y.narrow(d, 0, m).addcmul_(self.w[a], x.narrow(d, 1, m), value=-1.0)
        return y

    def solve(self, b, tol=2e-14):
        """Jacobi-preconditioned conjugate gradients."""
        inv = torch.where(self.diag > 0, 1.0 / self.diag.clamp(min=1e-300), 0.0)
        x, r = torch.zeros_like(b), b.clone()
        z = inv * r
        p, rz, norm = z.clone(), (r * z).sum(), float(b.norm())
        for it in range(30000):
            q = self.apply(p)
            alpha = rz / (p * q).sum()
            x += alpha * p
            r -= alpha * q
            z = inv * r
            new = (r * z).sum()
            p = z + (new / rz) * p
            rz = new
            if it % 100 == 99:
                r_true = b - self.apply(x)
                if float(r.norm()) <= tol * norm or float(r_true.norm()) <= tol * norm:
                    break
        return x

    def project(self, u, p, dt):
        div = torch.zeros_like(p)
        for a in range(3):
            div += (u[a].narrow(2 - a, 1, self.n[a]) - u[a].narrow(2 - a, 0, self.n[a])) / self.dx
        phi = self.solve(torch.where(self.fluid, -div / dt, 0.0))
        return [u[a] - dt * self.gradient(a, phi) for a in range(3)], p + phi

    def gradient(self, a, x):
        lo, hi = self.lohi(a, x)
        k = self.kind[a]
        g = torch.where(k == INTERIOR, (hi - lo) / self.dx, 0.0)
        return torch.where(k == OUTLET, (hi - lo) / (0.5 * self.dx), g)


# ------------------------------------------------------------------ inputs
def _uniform(shape, gen, lo=-1.0, hi=1.0):
    return torch.rand(shape, dtype=F64, device=DEV, generator=gen) * (hi - lo) + lo


def _flow_inputs(case, topo, site, seed):
    """Face velocities before a projection, and the pressure at hand."""
    gen = torch.Generator(device=DEV)
    gen.manual_seed(seed)
    noise = [_uniform(k.shape, gen) for k in topo.kind]
    if case["kind"] == "serve":  # the wind profile and a time step's disturbance
        u = [v + 0.05 * f for v, f in zip(topo.vel, noise)]
    elif case["kind"] == "step":  # the inflow and disturbances of a tenth of it
        u = [v + 0.1 * site["inflow"] * f for v, f in zip(topo.vel, noise)]
    else:
        u = noise
    p = torch.where(topo.fluid, _uniform(topo.fluid.shape, gen), 0.0)
    return topo.fixed(u), p


def _scalar_inputs(case, topo, site, seed):
    """Velocities, a plume, diffusivities, release densities, the time step and receptor weights."""
    gen = torch.Generator(device=DEV)
    gen.manual_seed(seed)
    u = topo.fixed([v + 0.1 * site["inflow"] * _uniform(k.shape, gen) for v, k in zip(topo.vel, topo.kind)])
    nz, ny, nx = topo.fluid.shape
    x = (torch.arange(nx, dtype=F64, device=DEV) + 0.5) / nx
    y = (torch.arange(ny, dtype=F64, device=DEV).reshape(-1, 1) + 0.5) / ny - 0.5
    z = (torch.arange(nz, dtype=F64, device=DEV).reshape(-1, 1, 1) + 0.5) / nz
    plume = 1e-3 * torch.exp(-(y / (0.05 + 0.3 * x)) ** 2 - (z / (0.1 + 0.5 * x)) ** 2)
    c = torch.where(topo.fluid, plume * _uniform(topo.fluid.shape, gen, 0.5, 1.0), 0.0)
    diff = torch.where(topo.fluid, _uniform(topo.fluid.shape, gen, 0.05, 0.15), 0.0)
    cells = torch.nonzero(topo.fluid.reshape(-1)).reshape(-1)
    at = cells[torch.randint(0, cells.numel(), (64,), device=DEV, generator=gen)]
    source = torch.zeros(topo.fluid.numel(), dtype=F64, device=DEV)
    source[at] = 1e-4
    dt = 0.4 * topo.dx / (2.0 * site["inflow"])
    rng = np.random.default_rng(case["receptors"])  # receptors are the site's: the same for every seed
    host = topo.fluid.reshape(-1).nonzero().reshape(-1).cpu().numpy()
    weights = [[(int(i), 0.125) for i in rng.choice(host, 8)] for _ in range(case["receptors"])]
    return u, c, diff, source.reshape(topo.fluid.shape), dt, weights


def _solve_inputs(case, seed):
    """A rough pressure without a mean, and its image under the operator."""
    n = _shape(case["cells"])
    gen = torch.Generator(device=DEV)
    gen.manual_seed(seed)
    i = torch.arange(n[0] * n[1] * n[2], dtype=F64, device=DEV).reshape(n[2], n[1], n[0])
    x = torch.sin(0.73 * i) + 0.3 * torch.cos(0.17 * i) + 0.1 * _uniform(i.shape, gen)
    x -= x.mean()
    size = (1.0, 1.0, case["thin"])
    b = torch.zeros_like(x)
    for a in (0, 2):
        d, w = 2 - a, (n[a] / size[a]) ** 2
        flux = w * (x.narrow(d, 1, n[a] - 1) - x.narrow(d, 0, n[a] - 1))
        b.narrow(d, 0, n[a] - 1).sub_(flux)
        b.narrow(d, 1, n[a] - 1).add_(flux)
    w = (n[1] / size[1]) ** 2
    b += w * (2.0 * x - torch.roll(x, 1, 1) - torch.roll(x, -1, 1))
    return x, b


# ------------------------------------------------------------------ what a program keeps
# A program opens its grids once and brings new inputs to them: the handles of the case at hand
# are kept from one preparation to the next, those of an earlier case are closed.
_open = {"key": None, "program": None}


def _program(case):
    key = json.dumps({k: v for k, v in case.items() if k != "name"}, sort_keys=True)
    if _open["key"] == key:
        return _open["program"]
    if _open["program"]:
        for h in reversed(_open["program"]["handles"]):
            h.close()
    _open.update(key=None, program=None)
    stream = torch.cuda.Stream()
    P = pkg.pressure
    if case["kind"] == "solve":
        grid = pkg.grid.Grid.build(_thin_case(case))
        prog = {"stream": stream, "handles": [P.DeviceGrid(grid, preconditioner="multigrid")]}
        prog["handles"][0].set_stream(stream.cuda_stream)
        _open.update(key=key, program=prog)
        return prog
    sites = _sites(case)
    form = {"batch": "mixed", "serve": "mixed", "scalar": "multigrid"}.get(case["kind"]) or case["form"]
    pre, precision = ("multigrid", "mixed") if form == "mixed" else (form, "plain")
    with ThreadPoolExecutor(max_workers=8) as ex:
        cases = [_framework_case(s, pre) for s in sites]
        grids = list(ex.map(pkg.grid.Grid.build, cases))
        topos = [Topo(s) for s in sites]
    handles = []
    for c, g in zip(cases, grids):
        d = P.DeviceGrid(g, preconditioner=pre, precision=precision)
        d.set_stream(stream.cuda_stream)
        if case["kind"] == "step":
            d.set_flow(c)
        handles.append(d)
    prog = {"stream": stream, "handles": handles, "sites": sites, "topos": topos}
    if case["kind"] == "batch":
        prog["batch"] = P.Batch(handles)
    elif case["kind"] == "serve":
        prog["batch"] = P.Server(handles, max_active=len(handles))
    elif case["kind"] == "scalar":
        handles[0].set_advection("muscl" if case["muscl"] else "linear_upwind")
        handles[0].set_receptors(_scalar_inputs(case, topos[0], sites[0], 0)[5])
    if "batch" in prog:
        prog["batch"].set_stream(stream.cuda_stream)
        handles.append(prog["batch"])
    _open.update(key=key, program=prog)
    return prog


def prepare(case, seed):
    prog = _program(case)
    s = {"case": case, "program": prog, "stream": prog["stream"], "grid": prog["handles"][0]}
    kind = case["kind"]
    if kind == "solve":
        s["b"] = _solve_inputs(case, seed)[1].reshape(-1).cpu().numpy()
    elif kind == "scalar":
        u, c, diff, source, dt, _ = _scalar_inputs(case, prog["topos"][0], prog["sites"][0], seed)
        s.update(u=Topo.flat(u), c=c.reshape(-1), diff=diff.reshape(-1), source=source.reshape(-1), dt=dt,
                 budget=torch.zeros(3, dtype=F64, device=DEV),
                 values=torch.empty(case["receptors"], dtype=F64, device=DEV))
    else:
        fields = [_flow_inputs(case, t, site, 1009 * seed + i) for i, (t, site) in enumerate(zip(prog["topos"], prog["sites"]))]
        s["u0"], s["p0"] = [Topo.flat(u) for u, _ in fields], [p.reshape(-1).contiguous() for _, p in fields]
        if kind == "serve":  # the fields of a served case stay in page-locked host memory
            for k in ("u0", "p0"):
                s[k] = [v.cpu().pin_memory() for v in s[k]]
            s["u"], s["p"] = ([torch.empty_like(v).pin_memory() for v in s[k]] for k in ("u0", "p0"))
        else:
            s["u"], s["p"] = [torch.empty_like(v) for v in s["u0"]], [torch.empty_like(v) for v in s["p0"]]
    torch.cuda.synchronize()  # the engine works on the program's own stream
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    with torch.cuda.stream(s["stream"]):
        if kind == "solve":
            x, _ = s["grid"].solve_scaled(s["b"], None, 1e-14, 1200)
            return {"x": x}
        if kind == "scalar":
            g, ptr = s["grid"], [s[k].data_ptr() for k in ("u", "c", "diff", "source")]
            if case["muscl"]:
                g.scalar_step_budget(*ptr, s["dt"], s["budget"].data_ptr())
            else:
                g.scalar_step_device(*ptr, s["dt"])
            g.sample_receptors(ptr[1], s["values"].data_ptr())
            out = {"c": s["c"], "values": s["values"]}
            return {**out, "budget": s["budget"]} if case["muscl"] else out
        u, p = [v.data_ptr() for v in s["u"]], [v.data_ptr() for v in s["p"]]
        if kind == "serve":
            server = s["program"]["batch"]
            left = [server.submit_host(i, s["u0"][i].data_ptr(), s["p0"][i].data_ptr(), u[i], p[i], case["dt"], TOL, MAX_ITER)
                    for i in range(len(u))]
            while left:
                server.progress()
                left = [t for t in left if _pending(server, t)]
        else:
            for k in ("u", "p"):
                for work, given in zip(s[k], s[k + "0"]):
                    work.copy_(given)
            if kind == "project":
                s["grid"].project_device(u[0], p[0], case["dt"], TOL, MAX_ITER)
            elif kind == "step":
                s["grid"].step_device(u[0], p[0], case["dt"], TOL, MAX_ITER)
            else:
                done = s["program"]["batch"].project_device(u, p, [case["dt"]] * len(u), TOL, MAX_ITER)
                if any(code for code, _ in done):
                    raise RuntimeError("a case of the batch failed")
    return {"u": s["u"], "p": s["p"]}


def _pending(server, ticket):
    r = server.result(ticket)
    if r is not None and r[0]:
        raise RuntimeError("a served request failed")
    return r is None


def work(case):
    if case["kind"] == "solve":
        nx, ny, nz = _shape(case["cells"])
        return {"bytes": 16.0 * nx * ny * nz, "flops": 13.0 * nx * ny * nz}
    total = {"bytes": 0.0, "flops": 0.0}
    for s in _sites(case):
        nx, ny, nz = s["cells"]
        N = nx * ny * nz
        F = (nx + 1) * ny * nz + nx * (ny + 1) * nz + nx * ny * (nz + 1)
        if case["kind"] == "scalar":  # u, c, diffusivity, release in; c out; two stages of flux sums
            total["bytes"] += 8.0 * F + 32.0 * N
            total["flops"] += 2.0 * (8.0 * 3 + 4.0) * N
        else:  # u and p in and out; right-hand side, operator, correction at least once
            total["bytes"] += 16.0 * F + 16.0 * N
            total["flops"] += (7.0 + 13.0 + 9.0) * N
    return total


# ------------------------------------------------------------------ 64-bit values
def exact(case, seed):
    if case["kind"] == "solve":
        return {"x": _solve_inputs(case, seed)[0].reshape(-1)}
    sites = _sites(case)
    if case["kind"] == "scalar":
        topo = Topo(sites[0])
        u, c, diff, source, dt, weights = _scalar_inputs(case, topo, sites[0], seed)
        r1, b1 = _rates(topo, u, c, diff, source, case["muscl"])
        stage = c + dt * r1
        r2, b2 = _rates(topo, u, stage, diff, source, case["muscl"])
        c = 0.5 * (c + stage + dt * r2)
        flat = c.reshape(-1)
        values = torch.stack([sum(flat[i] * w for i, w in ws) for ws in weights])
        out = {"c": flat, "values": values}
        return {**out, "budget": 0.5 * dt * (b1 + b2)} if case["muscl"] else out
    us, ps = [], []
    for i, site in enumerate(sites):
        topo = Topo(site)
        u, p = _flow_inputs(case, topo, site, 1009 * seed + i)
        if case["kind"] == "step":
            u, p = _exact_step(topo, site, u, p, case["dt"])
        else:
            u, p = topo.project(u, p, case["dt"])
        us.append(Topo.flat(u))
        ps.append(p.reshape(-1))
    return {"u": us, "p": ps}


def _momentum(topo, site, u, p, dt):
    """u + dt (R(u) - grad p) of laminar flow with donor-cell advection, fixed faces set."""
    dx, nu, vel = topo.dx, 1.5e-5, (site["inflow"], 0.0, 0.0)
    cell = [torch.where(topo.fluid, 0.5 * (u[a].narrow(2 - a, 0, topo.n[a]) + u[a].narrow(2 - a, 1, topo.n[a])), 0.0) for a in range(3)]
    out = []
    for a in range(3):
        k, uf = topo.kind[a], u[a]
        solid = (k == WALL) | (k == BLOCKED)
        rhs = torch.zeros_like(uf)
        for d in range(3):
            lo, hi = topo.lohi(a, cell[d])
            v = torch.where(k == INTERIOR, 0.5 * (lo + hi), lo + hi)
            dim, n = 2 - d, uf.shape[2 - d]
            near = []
            for side in (-1, 1):
                if d == a:  # beyond the domain's ends the face's own value
                    end = uf.narrow(dim, 0 if side < 0 else n - 1, 1)
                    parts = [end, uf.narrow(dim, 0, n - 1)] if side < 0 else [uf.narrow(dim, 1, n - 1), end]
                    near.append(torch.cat(parts, dim))
                    continue
                first = uf.narrow(dim, 0 if side < 0 else n - 1, 1)
                if site["bnd"][d] == "open":
                    inward = vel[d] * side < -1e-12
                    edge = 2.0 * vel[a] - first if inward else first
                else:
                    edge = -first
                m = n - 1
                val, sol = (uf.narrow(dim, 0, m), solid.narrow(dim, 0, m)) if side < 0 else (uf.narrow(dim, 1, m), solid.narrow(dim, 1, m))
                own = uf.narrow(dim, 1, m) if side < 0 else uf.narrow(dim, 0, m)
                inner = torch.where(sol, -own, val)  # no slip at a solid neighbour
                near.append(torch.cat([edge, inner], dim) if side < 0 else torch.cat([inner, edge], dim))
            back, forth = uf - near[0], near[1] - uf
            rhs = rhs - v * torch.where(v >= 0, back, forth) / dx + nu * (forth - back) / dx ** 2
        out.append(uf + dt * (rhs - topo.gradient(a, p)))
    return topo.fixed(out)


def _exact_step(topo, site, u, p, dt):
    u1, p1 = topo.project(_momentum(topo, site, u, p, dt), p, dt)
    u2, p2 = topo.project(_momentum(topo, site, u1, p1, dt), p1, dt)
    return topo.fixed([0.5 * (a + b) for a, b in zip(u, u2)]), p2


def _minmod(a, b):
    return torch.where(a * b > 0, torch.sign(a) * torch.minimum(a.abs(), b.abs()), 0.0)


def _rates(topo, u, c, diff, source, muscl):
    """dc/dt of a constituent, and (emitted, inflow, outflow) in kg/s."""
    dx, volume, area = topo.dx, topo.dx ** 3, topo.dx ** 2
    rate = source.clone()
    inflow, outflow = torch.zeros((), dtype=F64, device=DEV), torch.zeros((), dtype=F64, device=DEV)
    for a in range(3):
        d, n, k = 2 - a, topo.n[a], topo.kind[a]
        lo, hi = topo.lohi(a, c)
        dl, dh = topo.lohi(a, diff)
        fl, fh = topo.lohi(a, topo.fluid.to(F64))
        donor_lo, donor_hi = lo, hi
        if muscl:
            inner = k == INTERIOR
            below = torch.where(inner.narrow(d, 0, n), lo.narrow(d, 0, n), c)
            above = torch.where(inner.narrow(d, 1, n), hi.narrow(d, 1, n), c)
            slope = _minmod(0.5 * (above - below), _minmod(2.0 * (c - below), 2.0 * (above - c)))
            sl, sh = topo.lohi(a, slope)
            donor_lo, donor_hi = lo + 0.5 * sl, hi - 0.5 * sh
        donor = torch.where(u[a] >= 0, donor_lo, donor_hi)
        d_face = torch.where(k == INTERIOR, 0.5 * (dl + dh), dl + dh)
        dist = torch.where(k == INTERIOR, dx, 0.5 * dx)
        spread = torch.where(k == OUTLET, 0.0, d_face * (lo - hi) / dist)
        live = (k == INTERIOR) | (k == INLET) | (k == OUTLET)
        flux = torch.where(live, (u[a] * donor + spread) * area, 0.0)
        rate = rate + torch.where(topo.fluid, flux.narrow(d, 0, n) - flux.narrow(d, 1, n), 0.0) / volume
        outward = torch.where(k == INTERIOR, 0.0, flux * (fl - fh))
        inflow = inflow + (-outward).clamp(min=0.0).sum()
        outflow = outflow + outward.clamp(min=0.0).sum()
    return rate, torch.stack([source.sum() * volume, inflow, outflow])
