"""The solves that are timed: seeded fields advanced through the package's public entry points.

A pass is what a program does with a field it holds on the GPU: upload it into a solver context it
keeps (device to device), run the preamble of the time loop, advance it a few Runge-Kutta steps and
copy the advanced field back.  The contexts (grid, device buffers, launch shapes) are kept between
passes as a solver program keeps them; the fields are made from the seed.

Two kinds of starting field, the two regimes a run of the hybrid scheme goes through:
  noise      the mean flow plus uniform grid-scale noise on the velocities, as the synthetic initial
             fields of the package have it: a start-up transient in which most faces are WENO faces
  developed  the mean flow plus smooth solenoidal modes and a little grid-scale noise: the state of
             a running simulation, a few per cent of scattered WENO faces among central ones
"""
import ctypes
import math
import os
import sys
import tempfile
from functools import lru_cache

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "streams-2_b200"))

import streams_b200 as sb  # noqa: E402
from streams_b200.cases import SYNTHETIC_CP_POLY, batch_mix, bl_ini, channel_ini, shock_angle_for  # noqa: E402

# An interior cell and time step moves at least 440 bytes: the state, the two Runge-Kutta registers
# and the sensor, once each per stage (the boxes' states exceed the L2 from about a million cells on)
BYTES_PER_CELL_STEP = 440.0
# operations of a WENO5 and of a sixth-order central face, counted through the scheme's scalar
# code, and of the pointwise and viscous work of a stage
WENO_FACE, CENTRAL_FACE, CELL_REST = 1791.0, 385.0, 350.0
WENO_SHARE = {"noise": 0.9, "developed": 0.08}
# grid-scale noise on the velocities over u0: the start-up amplitudes of the synthetic fields, and
# for the developed state the fraction of the grid's resolution (the root sum square of 1/dx, 1/dy,
# 1/dz, dy in the wall-resolved part) at which 5 to 15 % of the faces start as WENO faces
NOISE = {("noise", "channel"): 0.1, ("noise", "bl"): 0.05, ("developed", "channel"): 0.5, ("developed", "bl"): 0.3}


def listed():
    return [
        # the smallest boxes of tests and parameter scans: 12 thousand cells, bound by launches
        # and by the latency of one block
        case("channel_tiny", "channel", 32, 24, 16, steps=10, start="noise"),
        # the smallest served solve, driven step by step from the host as the solver's own loop
        # does with residual monitoring (compute_dt, rk_sync, compute_residual)
        case("channel_driven_mixed", "channel", 48, 48, 48, steps=8, start="developed", precision=1,
             mode="driven"),
        # the parity and CPU-baseline configuration
        case("channel_128x96x64", "channel", 128, 96, 64, steps=6, start="noise"),
        # odd sizes that fill no tile, with WENO-Z and Sutherland viscosity
        case("channel_ragged", "channel", 189, 77, 93, steps=4, start="noise", weno_version=1, visc_model=2),
        # the supersonic channel at its benchmark size, in both precisions and regimes
        case("channel_512", "channel", 512, 256, 256, steps=2, start="noise"),
        case("channel_512_mixed", "channel", 512, 256, 256, steps=1, start="developed", precision=1),
        # the spatially developing boundary layer at its benchmark size: its transient and its
        # developed state (recycling inflow, non-reflecting outflow and top)
        case("bl_1024", "bl", 1024, 256, 192, steps=2, start="noise"),
        case("bl_1024_developed", "bl", 1024, 256, 192, steps=2, start="developed"),
        # the shock / boundary-layer interaction at its benchmark size in the mixed form
        case("sbli_1024_mixed", "sbli", 1024, 256, 128, steps=2, start="noise", precision=1),
        # a boundary layer of odd sizes with running statistics sampled every other step
        case("bl_ragged_stats", "bl", 301, 119, 77, steps=4, start="developed", mode="stats"),
        # parameter studies: uneven channels advanced together by one graph of shared launches
        case("batch_8", "batch", boxes=8, mix=2024, steps=11, start="noise"),
        case("batch_12_mixed", "batch", boxes=12, mix=7, steps=11, start="developed", precision=1),
    ]


def case(name, flow, nx=0, ny=0, nz=0, *, steps, start, precision=0, mode="advance", **more):
    c = dict(name=name, flow=flow, nx=nx, ny=ny, nz=nz, steps=steps, start=start, precision=precision, mode=mode)
    c.update(more)
    return c


def draw(rng):
    """A case of the same ranges: 12 thousand to 50 million cells, any sizes, the schemes, gases and
    viscosity laws that the solver offers."""
    u = rng.random()
    start = rng.choice(["noise", "developed"])
    precision = rng.choice([0, 0, 1])
    if u < 0.15:
        boxes = rng.randint(3, 12)
        c = case("", "batch", boxes=boxes, mix=rng.randint(1, 10 ** 6), steps=rng.choice([11, 12, 21 if boxes < 9 else 12]),
                 start=start, precision=precision)
        del c["name"]
        return c
    flow = "channel" if u < 0.65 else ("bl" if u < 0.9 else "sbli")
    lo, hi = (12e3, 40e6) if flow == "channel" else (3e5, 50e6)
    cells = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    b = (cells / (4.0 if flow == "channel" else 6.0)) ** (1.0 / 3.0)
    nx = int(2 * b * rng.uniform(0.8, 1.25)) if flow == "channel" else int(4 * b * rng.uniform(0.8, 1.1))
    ny = max(48 if flow != "channel" else 16, int(b * rng.uniform(0.8, 1.2)))
    nz = max(12, int(cells / (nx * ny)))
    steps = 2 if cells > 4e6 else (4 if cells > 4e5 else 8)
    more = {}
    if flow == "channel":
        more["mach"] = round(rng.uniform(0.3, 2.0), 4)
        more["re_bulk"] = round(rng.uniform(2000.0, 6000.0), 2)
    v = rng.random()
    if v < 0.15:
        more["weno_version"] = 1
    elif v < 0.25:
        more.update(ep_order=8, weno_scheme=4)
    elif v < 0.3:
        more.update(ep_order=4, weno_scheme=2)
    elif v < 0.4:
        more["flux_splitting"] = 1
    elif v < 0.48 and precision == 0:
        more["gas"] = "polynomial"  # the thermally perfect gas
    if rng.random() < 0.25:
        more["visc_model"] = 2
    if rng.random() < 0.15:
        more["conservative_viscous"] = 0
    if flow == "channel" and rng.random() < 0.1:
        more["nkeep"] = rng.choice([-1, 2])
    mode = rng.choice(["advance", "advance", "driven", "stats"] if cells < 4e6 else ["advance"])
    c = case("", flow, nx, ny, nz, steps=steps, start=start, precision=precision, mode=mode, **more)
    del c["name"]
    return c


OPTIONS = ("mach", "re_bulk", "weno_version", "ep_order", "weno_scheme", "flux_splitting", "visc_model",
           "conservative_viscous", "nkeep")


def inputs_of(c):
    """The input files of a case's boxes: (ini text, kind of flow)."""
    if c["flow"] == "batch":
        out = []
        for b in batch_mix(c["boxes"], c["mix"]):
            out.append((channel_ini(b["nx"], b["ny"], b["nz"], mach=b["mach"], re_bulk=b["re_bulk"], amp=0.0), "channel"))
        return out
    kw = {k: c[k] for k in OPTIONS if k in c}
    if "gas" in c:
        kw["cp_poly"] = SYNTHETIC_CP_POLY
    if c["flow"] == "channel":
        return [(channel_ini(c["nx"], c["ny"], c["nz"], amp=0.0, **kw), "channel")]
    if c["flow"] == "sbli":
        kw.update(mach=2.28, shock_angle=round(shock_angle_for(2.28), 4))
    return [(bl_ini(c["nx"], c["ny"], c["nz"], amp=0.0, **kw), "bl")]


@lru_cache(maxsize=24)
def setup(ini):
    """Host set-up of an input file (grid, metrics, mean flow).  It depends on no seed: a program
    that solves many fields on one grid keeps it."""
    with tempfile.TemporaryDirectory() as d:
        return sb.Case(d, ini)


def coordinates(s):
    nx, ny, nz, ng = s.shape
    g = s.grid()
    return [np.ctypeslib.as_array(p, (n + 2 * ng,)).copy() for p, n in ((g.x, nx), (g.y, ny), (g.z, nz))]


def field_of(s, kind, start, gen):
    """The seeded field w[m, k, j, i] (ghosts included) of a set-up, on the GPU."""
    nx, ny, nz, ng = s.shape
    shape = (5, nz + 2 * ng, ny + 2 * ng, nx + 2 * ng)
    mean = np.ctypeslib.as_array(sb.lib.streams_b200_case_field(s._h), shape)
    w = torch.from_numpy(mean).to("cuda")
    u0 = s.info()["u0"]
    vel = torch.rand((3,) + shape[1:], generator=gen, device="cuda", dtype=torch.float64).mul_(2).sub_(1)
    amp = NOISE[start, kind] * u0
    if start == "developed":
        x, y, z = (torch.from_numpy(a).cuda() for a in coordinates(s))
        lx, lz = float(x[-1 - ng] - x[ng]) * nx / (nx - 1), float(z[-1 - ng] - z[ng]) * nz / (nz - 1)
        amp /= math.sqrt((nx / lx) ** 2 + (nz / lz) ** 2 + (ny * (0.5 if kind == "channel" else 0.3)) ** 2)
    vel.mul_(amp)
    if start == "developed":
        if kind == "channel":  # between the walls at -1 and 1
            g, gp = (1 - y * y) ** 2, -4 * y * (1 - y * y)
        else:  # inside the layer, whose inflow thickness is 1
            g, gp = y * y * torch.exp(-y * y), (2 * y - 2 * y ** 3) * torch.exp(-y * y)
        r = torch.rand((6, 6), generator=gen, device="cuda", dtype=torch.float64).cpu().tolist()
        for a, b, cc, ph, n, m in r:
            # the curl of (a, b, cc) g(y) sin(kx x + kz z + phase): no divergence
            kx = 2 * math.pi / lx * (1 + int(n * (6 if kind == "channel" else 20)))
            kz = 2 * math.pi / lz * (1 + int(m * 4))
            th = (kx * x)[None, :] + (kz * z)[:, None] + 2 * math.pi * ph
            sn, cs = torch.sin(th)[:, None, :], torch.cos(th)[:, None, :]
            q = 0.06 * u0 / math.hypot(kx, kz)
            a, b, cc = (q * (2 * v - 1) for v in (a, b, cc))
            gy, gpy = g[None, :, None], gp[None, :, None]
            vel[0] += cc * gpy * sn - b * kz * gy * cs
            vel[1] += (a * kz - cc * kx) * gy * cs
            vel[2] += b * kx * gy * cs - a * gpy * sn
    rho = w[0]
    for m in range(3):  # E gains rho (u.du + du.du/2)
        w[4] += vel[m] * (w[1 + m] + 0.5 * rho * vel[m])
        w[1 + m] += rho * vel[m]
    return w


class State:
    pass


def prepare(c, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    st = State()
    st.case = c
    st.solvers, st.fields, st.out = [], [], []
    for ini, kind in inputs_of(c):
        s = setup(ini)
        w = field_of(s, kind, c["start"], gen)
        st.solvers.append(sb.Solver(s.params(c["precision"]), s.grid(), keepalive=s))
        st.fields.append(w)
        st.out.append(torch.empty_like(w))
    st.batch = sb.Batch(st.solvers, steps_per_graph=10) if c["flow"] == "batch" else None
    torch.cuda.synchronize()
    return st


def upload(s, w):
    s._check(sb.lib.streams_b200_copy_from_device(s._h, ctypes.c_void_p(w.data_ptr())))
    s.init_run()


def download(s, w):
    s._check(sb.lib.streams_b200_copy_to_device(s._h, ctypes.c_void_p(w.data_ptr())))


def run(st):
    c = st.case
    for s, w in zip(st.solvers, st.fields):
        upload(s, w)
    out = {}
    if st.batch is not None:
        st.batch.advance(c["steps"])
    else:
        s = st.solvers[0]
        if c["mode"] == "driven":
            out["dt"], out["residual"] = [], []
            for _ in range(c["steps"]):
                out["dt"].append(s.compute_dt())
                s.rk_sync()
                out["residual"].append(s.compute_residual()["residual_rhou"])
        elif c["mode"] == "stats":
            s.set_stats(0, np.zeros(s._stats_shape(0)))
            for n in range(c["steps"]):
                s.advance(1)
                if n % 2:
                    s.compute_stats(n // 2)
            out["stats"] = s.stats(0)
        else:
            s.advance(c["steps"])
    for b, (s, w) in enumerate(zip(st.solvers, st.out)):
        download(s, w)
        for m, name in enumerate(("rho", "rhou", "rhov", "rhow", "rhoe")):
            out[f"{name}{b}"] = w[m]
    return out


def work(c):
    if c["flow"] == "batch":
        cells = sum(b["nx"] * b["ny"] * b["nz"] for b in batch_mix(c["boxes"], c["mix"]))
    else:
        cells = c["nx"] * c["ny"] * c["nz"]
    share = WENO_SHARE[c["start"]]
    flops = 3 * (3 * (share * WENO_FACE + (1 - share) * CENTRAL_FACE) + CELL_REST)
    # the field is read once and written once beside the steps
    return {"bytes": cells * (c["steps"] * BYTES_PER_CELL_STEP + 80.0), "flops": cells * c["steps"] * flops}


def tolerance(c):
    """FP64: the solver is 1e-15 (rho, rhou, rhoE) to 1.4e-14 (the transverse momenta, which are as
    small as the perturbations) from the 64-bit channel below after 2 to 11 steps, 1.1e-13 of the rms
    at the worst point; open boundaries and the gas with a Newton iteration get a margin on that.

    Mixed: without a point whose sensor crosses its threshold differently, 2.3e-6 and 2e-5 from the
    64-bit channel.  One that does switches a face between the WENO and the central flux, an O(1)
    change there, more of them in noise and with the steps: the mixed and the FP64 form were 7e-6
    (developed; 1.3e-5 another time), 7e-5 (noise, up to 4 steps) and 1.8e-3 (noise, 11 steps) apart,
    at the worst point 0.02, 0.1 and 0.4 of the rms."""
    if c["precision"] == 0:
        return {"rel": 5e-13, "max": 2e-11}
    if c["start"] == "developed":
        return {"rel": 6e-5, "max": 0.2}
    return {"rel": 3e-4, "max": 0.4} if c["steps"] <= 4 else {"rel": 7e-3, "max": 0.9}


# ---------------------------------------------------------------------------------------------
# The channel advanced in 64-bit torch, written from the scheme's formulas (no code of this
# repository): periodic x and z, staggered isothermal walls in y, sixth-order central / WENO5 with
# Roe splitting, conservative viscous form, bulk forcing with the bulk temperature held.

def exact(c, seed):
    if c["flow"] not in ("channel", "batch") or c["nx"] * c["ny"] * c["nz"] * c["steps"] > 8e7:
        return None  # open boundaries: the inflow continues the set-up's random sequence
    if c["precision"] == 1 and c["steps"] > 1 and work(c)["bytes"] > 1e9:
        return None  # about as many crossings of the sensor's threshold as FP32 rounding: see tolerance()
    if any(k in c for k in ("ep_order", "flux_splitting", "conservative_viscous", "nkeep", "gas")):
        return None
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    names = ("rho", "rhou", "rhov", "rhow", "rhoe")
    out = {}
    for b, (ini, kind) in enumerate(inputs_of(c)):
        s = setup(ini)
        w = field_of(s, kind, c["start"], gen)
        if b >= 2:  # two boxes of a batch; each takes about a second
            for n in names:
                out[f"{n}{b}"] = None
            continue
        ch = Channel(s)
        w, dts, res = ch.solve(w, c["steps"])
        for m, n in enumerate(names):
            out[f"{n}{b}"] = w[m]
        if c["mode"] == "driven":
            out["dt"], out["residual"] = dts, res
        if c["mode"] == "stats":
            out["stats"] = None
    return out


class Channel:
    COEFF = {3: (0.75, -0.15, 1.0 / 60.0), 2: (2.0 / 3.0, -1.0 / 12.0), 1: (0.5,)}

    def __init__(self, s):
        p, g = s.params(0), s.grid()
        self.p, self.ng = p, p.ng
        self.n = (p.nx, p.ny, p.nz)

        def arr(ptr, n):
            return torch.from_numpy(np.ctypeslib.as_array(ptr, (n,)).copy()).cuda()
        self.x = [arr(q, n + 2 * p.ng) for q, n in zip((g.x, g.y, g.z), self.n)]
        self.dy = arr(g.yn, p.ny + 1).diff().view(1, -1, 1)
        self.met = [arr(q, n) for q, n in zip((g.dcsidx, g.detady, g.dzitdz), self.n)]
        self.met2 = [arr(q, n) for q, n in zip((g.dcsidxs, g.detadys, g.dzitdzs), self.n)]
        self.gam = p.cp0 / (p.cp0 - p.rgas0)

    # a vector along direction d as a (z, y, x) broadcast
    def along(self, v, d):
        return v.view([-1 if 2 - a == d else 1 for a in range(3)])

    # the interior of a ghosted array, shifted by o points
    def at(self, a, o=(0, 0, 0)):
        g = self.ng
        i, j, k = (slice(g + o[d], g + o[d] + self.n[d]) for d in range(3))
        return a[..., k, j, i]

    def temperature(self, w):
        rho = w[0]
        u = w[1:4] / rho
        ee = w[4] / rho - 0.5 * (u * u).sum(0)
        return self.p.t0 + (ee - self.p.cv_last * self.p.t0) / self.p.cv0

    def energy(self, t):
        return (self.p.cv_last + self.p.cv0 * (t / self.p.t0 - 1.0)) * self.p.t0

    def fill(self, w):
        """Face ghosts: periodic copies in x and z, mirrored states at the isothermal walls."""
        g, (nx, ny, nz) = self.ng, self.n
        I, J, K = slice(g, g + nx), slice(g, g + ny), slice(g, g + nz)
        w[:, K, J, :g], w[:, K, J, g + nx:] = w[:, K, J, nx:nx + g].clone(), w[:, K, J, g:2 * g].clone()
        w[:, :g, J, I], w[:, g + nz:, J, I] = w[:, nz:nz + g, J, I].clone(), w[:, g:2 * g, J, I].clone()
        for dst, src in ((slice(0, g), slice(g, 2 * g)), (slice(g + ny, None), slice(ny, g + ny))):
            q = w[:, K, src, I].flip(2)
            t = self.temperature(q)
            pp = q[0] * t * self.p.rgas0
            u = q[1:4] / q[0]
            tg = 2.0 * self.p.t_wall - t
            rho = pp / tg / self.p.rgas0
            w[0, K, dst, I] = rho
            w[1:4, K, dst, I] = -rho * u
            w[4, K, dst, I] = rho * (self.energy(tg) + 0.5 * (u * u).sum(0))

    def aux(self, w):
        """rho, u, v, w, H, T, mu at all points (edges and corners hold what w has there)."""
        self.fill(w)
        a = torch.empty((7,) + w.shape[1:], dtype=w.dtype, device=w.device)
        a[0] = w[0]
        a[1:4] = w[1:4] / w[0]
        t = self.temperature(w)
        a[5] = t
        a[4] = (w[4] + w[0] * t * self.p.rgas0) / w[0]
        tr = t / self.p.t0
        if self.p.visc_model == 1:
            a[6] = self.p.mu0 * tr.abs() ** self.p.powerlaw_vtexp
        else:
            q = self.p.sutherland_s / self.p.t_ref_dim
            a[6] = self.p.mu0 * tr.abs() ** 1.5 * (1.0 + q) / (tr + q)
        return a

    def grads(self, a):
        """[d][f]: second-order derivatives of u, v, w, T, mu along d."""
        out = []
        for d in range(3):
            x, g, n = self.x[d], self.ng, self.n[d]
            r = self.along(1.0 / (x[g + 1:g + n + 1] - x[g - 1:g + n - 1]), d)
            o = [0, 0, 0]
            o[d] = 1
            hi, lo = self.at(a, o), self.at(a, [-v for v in o])
            out.append([r * (hi[f] - lo[f]) for f in (1, 2, 3, 5, 6)])
        return out

    def sensor(self, gr):
        div = gr[0][0] + gr[1][1] + gr[2][2]
        om = (gr[1][2] - gr[2][1]) ** 2 + (gr[2][0] - gr[0][2]) ** 2 + (gr[0][1] - gr[1][0]) ** 2
        q = self.p.u0 / self.p.l0
        return torch.clamp(-div / torch.sqrt(om + div * div + q * q), min=0.0) ** 2

    def time_step(self, a):
        q = self.at(a)
        cs = torch.sqrt(self.gam * self.p.rgas0 * q[5])
        nu = q[6] / q[0]
        most = 0.0
        for d in range(3):
            m, m2 = self.along(self.met[d], d), self.along(self.met2[d], d)
            for v in ((q[1 + d].abs() + cs) * m, nu * m2, nu / self.p.prandtl * m2):
                most = max(most, float(v.max()))
        return self.p.cfl / most

    def pad(self, s):
        """The interior sensor with 3 ghost layers: periodic in x and z, 0 beyond the walls."""
        s = torch.nn.functional.pad(s, (0, 0, 3, 3))
        s = torch.cat([s[:, :, -3:], s, s[:, :, :3]], 2)
        return torch.cat([s[-3:], s, s[:3]], 0)

    def faces(self, a, sens, d):
        """Divergence of the hybrid face fluxes along d; slabs bound the temporaries."""
        g, n = self.ng, self.n
        t = 2 if d != 2 else 1  # the direction that is cut into slabs
        other = [e for e in range(3) if e != d]
        per = max(1, int(3e6 / (n[d] * n[3 - d - t])))
        out = torch.empty((5,) + tuple(reversed(n)), dtype=a.dtype, device=a.device)
        flag = sens > self.p.sensor_threshold
        ax = {0: 3, 1: 2, 2: 1}
        for b in range(0, n[t], per):
            e = min(n[t], b + per)
            q = a[:6].narrow(ax[t], g + b, e - b).narrow(ax[3 - d - t], g, n[3 - d - t]).movedim(ax[d], 1)
            f = flag.narrow(ax[t] - 1, 3 + b, e - b).narrow(ax[3 - d - t] - 1, 3, n[3 - d - t]).movedim(ax[d] - 1, 0)
            nf = n[d] + 1  # face p between the points p and p+1: its stencil is p-2 .. p+3
            st = [q[:, g - 3 + o:g - 3 + o + nf] for o in range(6)]
            weno = f[0:nf].clone()
            for o in range(1, 6):
                weno |= f[o:o + nf]
            fl = torch.empty((5,) + tuple(weno.shape), dtype=a.dtype, device=a.device)
            for lo, hi, order in self.orders(d, nf):
                part = [p[:, lo:hi] for p in st]
                wf = weno[lo:hi]
                c = self.central(part, d, order)
                if order < 3 and d == 1 and lo in (0, nf - 1):  # no convective flux through a wall
                    c = torch.zeros_like(c)
                    c[1 + d] = self.central(part, d, order, pressure=True)
                fl[:, lo:hi] = torch.where(wf, self.weno(part, d, order), c)
            div = (fl[:, 1:] - fl[:, :-1]) * self.met[d].view(1, -1, 1, 1)
            out.narrow(ax[t], b, e - b).copy_(div.movedim(1, ax[d]))
        return out

    def orders(self, d, nf):
        """(first face, past the last, half order): 1, 1, 2 next to a wall, 3 elsewhere."""
        if d != 1:
            return [(0, nf, 3)]
        return [(0, 1, 1), (1, 2, 1), (2, 3, 2), (3, nf - 3, 3), (nf - 3, nf - 2, 2), (nf - 2, nf - 1, 1), (nf - 1, nf, 1)]

    def central(self, st, d, order, pressure=False):
        R = self.p.rgas0
        pp = [q[0] * q[5] * R for q in st]
        ee = [q[4] - q[5] * R - 0.5 * (q[1] ** 2 + q[2] ** 2 + q[3] ** 2) for q in st]
        f = [0.0] * 5
        f6 = 0.0
        for l in range(1, order + 1):
            s = [0.0] * 5
            s6 = 0.0
            for m in range(l):
                a, b = 2 - m, 2 - m + l
                A, B = st[a], st[b]
                uv = (A[1 + d] + B[1 + d]) * (A[0] + B[0])
                s[0] = s[0] + 2 * uv
                for v in range(3):
                    s[1 + v] = s[1 + v] + uv * (A[1 + v] + B[1 + v])
                s[4] = s[4] + uv * (ee[a] + ee[b] + A[1] * B[1] + A[2] * B[2] + A[3] * B[3]) \
                    + 4 * (A[1 + d] * pp[b] + B[1 + d] * pp[a])
                s6 = s6 + 2 * (pp[a] + pp[b])
            cl = self.COEFF[order][l - 1]
            f = [x + cl * y for x, y in zip(f, s)]
            f6 = f6 + cl * s6
        if pressure:
            return 0.5 * f6
        f = [0.25 * x for x in f]
        f[1 + d] = f[1 + d] + 0.5 * f6
        return torch.stack(f)

    def weno(self, st, d, order):
        p, R = self.p, self.p.rgas0
        A, B = st[2], st[3]
        r = torch.sqrt(B[0] / A[0])
        ub = [(r * B[m] + A[m]) / (r + 1) for m in (1, 2, 3)]
        h = (r * B[4] + A[4]) / (r + 1)
        qq = 0.5 * (ub[0] ** 2 + ub[1] ** 2 + ub[2] ** 2)
        tt = p.t0 + (h - qq - p.cp_last * p.t0) / p.cp0
        c2 = self.gam * tt * R
        c = torch.sqrt(c2)
        b2 = (self.gam - 1) / c2
        et = h - tt * R
        b1 = tt * R / c2 - b2 * (et - 2 * qq)
        b3 = et - tt * R / (self.gam - 1)
        vn = ub[d]
        t1, t2 = [e for e in range(3) if e != d]
        cs = [torch.sqrt(self.gam * R * q[5]) for q in st]

        def most(v):
            return torch.stack(v).amax(0)
        lam = [most([(q[1 + d] - s).abs() for q, s in zip(st, cs)]), most([q[1 + d].abs() for q in st]), None, None,
               most([(q[1 + d] + s).abs() for q, s in zip(st, cs)])]
        lam[2] = lam[3] = lam[1]

        def project(X):
            s = b1 * X[0] + b2 * (X[4] - ub[0] * X[1] - ub[1] * X[2] - ub[2] * X[3])
            a = (vn * X[0] - X[1 + d]) / c
            return [0.5 * (s + a), X[0] - s, X[1 + t1] - ub[t1] * X[0], X[1 + t2] - ub[t2] * X[0], 0.5 * (s - a)]
        gp, gm = [[] for _ in range(5)], [[] for _ in range(5)]
        for q in st:
            pp = q[0] * q[5] * R
            U = [q[0], q[0] * q[1], q[0] * q[2], q[0] * q[3], q[0] * q[4] - pp]
            F = [q[0] * q[1 + d] * v for v in (1.0, q[1], q[2], q[3], q[4])]
            F[1 + d] = F[1 + d] + pp
            PU, PF = project(U), project(F)
            for m in range(5):
                gp[m].append(0.5 * (PF[m] + lam[m] * PU[m]))
                gm[m].append(0.5 * (PF[m] - lam[m] * PU[m]))
        r2 = p.rho0 ** 2
        scale = [1 / (r2 * p.u0 ** 2)] * 2 + [1 / (r2 * p.u0 ** 4)] * 2 + [1 / (r2 * p.u0 ** 2)]
        fi = [self.rec(gp[m][:5], scale[m], order) + self.rec(gm[m][:0:-1], scale[m], order) for m in range(5)]
        f = [fi[0] + fi[1] + fi[4]]
        for e in range(3):
            v = ub[e] * f[0]
            if e == d:
                v = v + c * (fi[4] - fi[0])
            if e == t1:
                v = v + fi[2]
            if e == t2:
                v = v + fi[3]
            f.append(v)
        f.append((h - vn * c) * fi[0] + b3 * fi[1] + ub[t1] * fi[2] + ub[t2] * fi[3] + (h + vn * c) * fi[4])
        return torch.stack(f)

    def rec(self, v, scale, order):
        """Reconstruction at the face from v[0..4], the upwind point at v[2]."""
        if order == 1:
            return v[2]
        if order == 2:
            w = [d / (1e-6 + scale * (a - b) ** 2) ** 2
                 for d, a, b in ((1 / 3, v[2], v[1]), (2 / 3, v[3], v[2]))]
            return 0.5 * (w[0] * (3 * v[2] - v[1]) + w[1] * (v[2] + v[3])) / (w[0] + w[1])
        be = [13 / 12 * (v[0] - 2 * v[1] + v[2]) ** 2 + 0.25 * (v[0] - 4 * v[1] + 3 * v[2]) ** 2,
              13 / 12 * (v[1] - 2 * v[2] + v[3]) ** 2 + 0.25 * (v[1] - v[3]) ** 2,
              13 / 12 * (v[2] - 2 * v[3] + v[4]) ** 2 + 0.25 * (3 * v[2] - 4 * v[3] + v[4]) ** 2]
        be = [scale * b for b in be]
        if self.p.weno_version == 0:
            w = [d / (1e-6 + b) ** 2 for d, b in zip((0.1, 0.6, 0.3), be)]
        else:
            tiny = float(np.float32(1e-35))
            tau = (be[0] - be[2]).abs() + tiny
            w = [d * (b + tau) / (b + tiny) for d, b in zip((0.1, 0.6, 0.3), be)]
        q = [(2 * v[0] - 7 * v[1] + 11 * v[2]) / 6, (-v[1] + 5 * v[2] + 2 * v[3]) / 6, (2 * v[2] + 5 * v[3] - v[4]) / 6]
        return (w[0] * q[0] + w[1] * q[1] + w[2] * q[2]) / (w[0] + w[1] + w[2])

    def viscous(self, a, gr, div3):
        """What the viscous terms add to the convective divergence (momenta and energy)."""
        p, q = self.p, self.at(a)
        mg = [gr[d][4] for d in range(3)]
        sig = [[gr[i][j] - (2 * div3 if i == j else 0.0) for j in range(3)] for i in range(3)]
        f = torch.zeros((5,) + tuple(q.shape[1:]), dtype=a.dtype, device=a.device)
        s = [mg[0] * sig[j][0] + mg[1] * sig[j][1] + mg[2] * sig[j][2] for j in range(3)]
        heat = sum(sig[i][j] * gr[j][i] for i in range(3) for j in range(3))
        for j in range(3):
            f[1 + j] -= s[j]
            f[4] -= s[j] * q[1 + j]
        f[4] -= heat * q[6]
        for d in range(3):
            x, g, n = self.x[d], self.ng, self.n[d]
            o = [0, 0, 0]
            o[d] = 1
            pts = [self.at(a, [-v for v in o]), q, self.at(a, o)]
            xs = [x[g - 1 + e:g - 1 + e + n] for e in range(3)]
            hl = self.along(2.0 / (xs[2] - xs[0]), d)
            for sgn, L, U, xl, xu in ((1.0, pts[0], pts[1], xs[0], xs[1]), (-1.0, pts[1], pts[2], xs[1], xs[2])):
                mf = 0.5 * (L[6] + U[6]) / self.along(xu - xl, d)
                ke = 0.5 * (U[1] ** 2 + U[2] ** 2 + U[3] ** 2 - L[1] ** 2 - L[2] ** 2 - L[3] ** 2)
                for j in range(3):
                    f[1 + j] += sgn * hl * (U[1 + j] - L[1 + j]) * mf
                f[4] += sgn * hl * ((U[5] - L[5]) * p.cp0 / p.prandtl + ke) * mf
        for d in range(3):  # grad(mu div/3): div/3 periodic in x and z, nearest interior beyond a wall
            x, g, n = self.x[d], self.ng, self.n[d]
            r = self.along(1.0 / (x[g + 1:g + n + 1] - x[g - 1:g + n - 1]), d)
            dim = 2 - d
            up, dn = torch.roll(div3, -1, dim), torch.roll(div3, 1, dim)
            if d == 1:
                up[:, -1], dn[:, 0] = div3[:, -1], div3[:, 0]
            t = q[6] * r * (up - dn)
            f[1 + d] -= t
            f[4] -= t * q[1 + d]
        return f

    def solve(self, w, steps):
        p = self.p
        w = w.clone()
        inner = self.at(w)
        a = self.aux(w)
        sens = self.sensor(self.grads(a))
        prev, shift, dts, res = None, None, [], []
        fv = p.channel_case and p.theta_wall >= -1.0
        for _ in range(steps):
            for stage in range(3):
                if shift is not None:
                    t = self.temperature(inner) + shift
                    inner[4] = inner[0] * self.energy(t) + 0.5 * (inner[1] ** 2 + inner[2] ** 2 + inner[3] ** 2) / inner[0]
                    shift = None
                a = self.aux(w)
                if stage == 0:
                    dt = self.time_step(a)
                    dts.append(dt)
                gr = self.grads(a)
                div3 = (gr[0][0] + gr[1][1] + gr[2][2]) / 3.0
                fl = self.viscous(a, gr, div3)
                for d in range(3):
                    fl += self.faces(a, self.pad(sens), d)
                if stage == 2:
                    sens = self.sensor(gr)
                fln = -p.gamrk[stage] * dt * fl
                if stage > 0:
                    fln -= p.rhork[stage] * dt * prev
                prev = fl
                b = [float((v * self.dy).sum()) / p.volchan for v in (fln[0], fln[1], inner[0], inner[1])]
                fln[0] -= b[0]
                fln[1] -= b[1]
                fln[4] -= inner[1] / inner[0] * b[1]
                inner += fln
                if fv:
                    t = self.temperature(inner)
                    shift = p.t_bulk_target - float((inner[1] * t * self.dy).sum()) / p.volchan / b[3]
            res.append(math.sqrt(float((fln[1] / dt).square().mean())))
        if shift is not None:
            t = self.temperature(inner) + shift
            inner[4] = inner[0] * self.energy(t) + 0.5 * (inner[1] ** 2 + inner[2] ** 2 + inner[3] ** 2) / inner[0]
        self.fill(w)
        return w, dts, res
