"""The work a user of this package has it do, as timed cases through its public entry points.

Every case is a problem preset with its grid, scheme, Riemann solver and precision policy,
and a way of calling the library:

``step``   the drop-in calls of a driver that keeps its own time loop on the host: upload
           the conserved state, con2prim, the CFL step, one SSP-RK3 step, download.
``solve``  a short solve from host data: upload, prim_to_cons, the time loop, download.
``run``    one resident grid advanced by the time loop, its state copied out afterwards.
``rhs``    the spatial operator alone: upload primitives, right-hand side to the host.
``batch``  many equal resident grids stepped together (graph replays, autotuned), states
           copied out afterwards.
``serve``  a batch of uneven 1D requests of the serving stream, states copied out.
``e2e``    equal grids in sub-batches on their own streams; every step uploads each grid's
           conserved state from page-locked memory, recovers the primitives, steps, and
           downloads the state.

``exact`` restates the whole path in plain 64-bit torch from the host set-up's metric
tables and initial data.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from grhd_b200 import native as N
from grhd_b200.problem import Problem
from grhd_b200.serve import make_stream
from grhd_b200.solver import GpuBatch, GpuGrid

FM = dict(metric="kerr_schild", geometry="spheroidal", logarithmic_r=True, spin=0.9, bh_mass=1.0, r_min=1.2,
          r_max=40.0, theta_min=0, theta_max=1, phi_min=0, phi_max=2, fm_inner_radius=6.0,
          fm_pressure_max_radius=12.0, fm_polytropic_constant=0.0015, adiabatic_index=1.3333333333333333, cfl=0.4,
          perturbation="pressure_noise", perturbation_amplitude=0.01, perturbation_time=0.0)
PRESETS = {
    # relativistic blast wave on x in [0, 1]
    "sod": dict(adiabatic_index=1.6666666666666667, sod_interface=0.5, sod_density_left=10, sod_pressure_left=13.33,
                sod_density_right=1, sod_pressure_right=1e-6, cfl=0.4, final_time=0.4,
                perturbation="pressure_noise", perturbation_amplitude=0.01, perturbation_time=0.0),
    "kelvin_helmholtz": dict(perturbation="pressure_noise", perturbation_amplitude=0.01, perturbation_time=0.0),
    # accretion onto Schwarzschild, ingoing Eddington-Finkelstein, log r
    "michel": dict(metric="eddington_finkelstein", geometry="spherical", logarithmic_r=True, bh_mass=1.0, r_min=1.8,
                   r_max=20.0, adiabatic_index=1.3333333333333333, michel_critical_radius=8.0, final_time=500.0,
                   perturbation="density_noise", perturbation_amplitude=0.001, perturbation_time=0.0),
    # Fishbone-Moncrief tori in Kerr-Schild coordinates
    "fishbone_equatorial": FM, "fishbone_sagittal": FM, "fishbone_3d": FM,
}


def _case(name, call, problem, nx, ny=1, nz=1, rec="weno5", rs="hlle", sensor=False, precision="fp64", grids=1, steps=1,
          stream=0):
    c = dict(call=call, problem=problem, nx=nx, ny=ny, nz=nz, rec=rec, rs=rs, sensor=sensor, precision=precision,
             grids=grids, steps=steps, stream=stream)
    return dict(c, name=name) if name else c


def listed():
    return [
        # one host-driven step of a small odd-sized Riemann problem: nothing but latency
        _case("sod_131_step", "step", "sod", 131, rec="mp5", rs="hllc"),
        # the shock-tube configuration, a short solve from host data
        _case("sod_400_solve", "solve", "sod", 400, steps=20),
        # the Michel accretion configuration, resident, under the mixed policy
        _case("michel_1024_mixed_run", "run", "michel", 1024, rec="mp5", precision="mixed", steps=20),
        # a server's resident batch: uneven Riemann problems and Michel runs
        _case("serve_64_fp64", "serve", "sod", 0, grids=64, steps=6, stream=20260901),
        _case("serve_64_mixed", "serve", "sod", 0, grids=64, steps=6, stream=20260902, precision="mixed"),
        # the spatial operator of a ragged x-y torus (the fine-grained entry of a host driver)
        _case("sagittal_257x131_rhs", "rhs", "fishbone_sagittal", 257, ny=131, rec="weno3"),
        # one 2.5D torus alone, and the headline batch of 32 in both precisions
        _case("torus2p5d_run", "run", "fishbone_equatorial", 400, nz=200, steps=10),
        _case("torus2p5d_x32_fp64", "batch", "fishbone_equatorial", 400, nz=200, grids=32, steps=4),
        _case("torus2p5d_x32_mixed", "batch", "fishbone_equatorial", 400, nz=200, grids=32, steps=4, precision="mixed"),
        # states that live on the host: 16 tori uploaded, recovered, stepped and downloaded
        _case("torus2p5d_x16_e2e", "e2e", "fishbone_equatorial", 400, nz=200, grids=16, steps=1),
        # the 3D torus configuration in both precisions
        _case("torus3d_fp64_run", "run", "fishbone_3d", 256, 128, 128, "mp5", "hllc", True, steps=2),
        _case("torus3d_mixed_run", "run", "fishbone_3d", 256, 128, 128, "mp5", "hllc", True, "mixed", steps=2),
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    call = rng.choice(("step", "solve", "run", "serve", "rhs", "batch", "batch", "e2e", "run"))
    prec = rng.choice(("fp64", "fp64", "mixed", "mixed", "mixed_comp64"))
    rs = rng.choice(("hlle", "hlle", "hllc"))
    wide = rng.choice(("weno5", "mp5"))  # three ghost cells; the shock sensor goes with these
    sensor = rng.random() < 0.3
    if call in ("step", "solve"):
        if rng.random() < 0.7:
            return _case("", call, "sod", log(128, 8192), rec=rng.choice(("weno5", "mp5", "weno3", "tvd")), rs=rs,
                         precision=prec, steps=1 if call == "step" else rng.randint(5, 30))
        return _case("", call, "kelvin_helmholtz", log(48, 500), nz=log(48, 300), rec=wide, rs=rs, sensor=sensor,
                     precision=prec, steps=1 if call == "step" else rng.randint(2, 8))
    if call == "serve":
        return _case("", call, "sod", 0, grids=log(8, 64), steps=rng.randint(3, 6), stream=rng.randint(1, 10**6),
                     precision=rng.choice(("fp64", "mixed")))
    if call == "rhs":
        return _case("", call, "fishbone_sagittal", log(64, 500), ny=log(32, 300),
                     rec=rng.choice(("weno5", "mp5", "weno3", "tvd")), rs=rs, precision=rng.choice(("fp64", "fp64", "mixed")))
    if call == "batch":
        if rng.random() < 0.25:
            return _case("", call, "michel", log(256, 4096), rec="mp5", rs=rs, precision=prec, grids=log(4, 48),
                         steps=rng.randint(2, 4))
        return _case("", call, "fishbone_equatorial", log(64, 400), nz=log(32, 200), rec=wide, rs=rs, sensor=sensor,
                     precision=prec, grids=log(2, 32), steps=rng.randint(2, 4))
    if call == "e2e":
        return _case("", call, "fishbone_equatorial", log(64, 400), nz=log(32, 200), rec=wide, rs=rs,
                     precision=rng.choice(("fp64", "mixed")), grids=log(4, 16), steps=1)
    which = rng.random()
    if which < 0.25:
        return _case("", call, "michel", log(256, 4096), rec=wide, rs=rs, precision=prec, steps=rng.randint(5, 20))
    if which < 0.6:
        return _case("", call, "fishbone_equatorial", log(64, 600), nz=log(32, 300), rec=wide, rs=rs, sensor=sensor,
                     precision=prec, steps=rng.randint(3, 10))
    return _case("", call, "fishbone_3d", log(32, 200), log(16, 128), 2 * log(8, 64), wide, rs, sensor, prec,
                 steps=rng.randint(1, 2))


# ---- what a user's program has in hand -----------------------------------------------------
def _problems(c, seed):
    """The problems of a case; the seed sets the perturbation noise of each grid."""
    base = 1 + 1000 * (seed % 1_000_000)
    if c["call"] == "serve":
        out = []
        for q, r in enumerate(make_stream(n=c["grids"], seed=c["stream"])):
            noise = "density_noise" if r.kind == "michel" else "pressure_noise"
            out.append(Problem.from_keys(r.problem, **dict(r.keys, perturbation=noise, perturbation_amplitude=0.001,
                                                           perturbation_time=0.0, perturbation_seed=base + q)))
        return out
    keys = dict(PRESETS[c["problem"]], nx=c["nx"], ny=c["ny"], nz=c["nz"], reconstruction=c["rec"],
                riemann_solver=c["rs"], shock_sensor=c["sensor"])
    return [Problem.from_keys(c["problem"], **dict(keys, perturbation_seed=base + q)) for q in range(c["grids"])]


def _initial(pb):
    p = pb.initial_prims()
    pb.perturb(p)
    return p


def _grid(pb, precision, stream=None):
    g = GpuGrid(pb, precision=precision, upload_initial=False, stream=stream.cuda_stream if stream else None)
    g.upload(p=_initial(pb))
    g.prim_to_cons()
    return g


def _pinned(pbs):
    """One page-locked conserved-state array per problem."""
    return [torch.empty(pb.cons_shape, dtype=torch.float64).pin_memory() for pb in pbs]


class _State:
    """Grids, batches and host buffers, released together (batches before their grids)."""

    def __init__(self, case):
        self.case, self.grids, self.batches = case, [], []

    def __del__(self):
        for x in self.batches + self.grids:
            x.close()


def prepare(case, seed):
    s = _State(case)
    pbs = _problems(case, seed)
    call, prec = case["call"], case["precision"]
    if call in ("step", "solve", "rhs"):
        s.grids = [_grid(pbs[0], prec)]
        s.p0 = _initial(pbs[0])
        s.up0 = s.grids[0].download(want_p=False)[0]
        s.dt = s.grids[0].cfl()
        return s
    if call == "run":
        s.grids = [_grid(pbs[0], prec)]
        s.out = _pinned(pbs)
    else:
        nsub = min(4, len(pbs)) if call == "e2e" else 1
        s.streams = [torch.cuda.Stream() for _ in range(nsub)]
        s.subs, s.out = [], []
        for q, st in enumerate(s.streams):
            grids = [_grid(pb, prec, st) for pb in pbs[q::nsub]]
            s.grids += grids
            out = _pinned(pbs[q::nsub])
            s.out += out
            b = GpuBatch(grids)
            s.batches.append(b)
            for k in range(len(grids)):
                b.set_clock(k, 0.0, 1e300, -1)
            if call in ("batch", "e2e"):
                b.autotune(reps=5)
            s.subs.append((b, grids, out))
        if call == "e2e":
            for g, o in zip(s.grids, s.out):
                o.numpy()[...] = g.download(want_p=False)[0]
    s.lib = s.grids[0].lib
    s.ptr = {id(o): N.dptr(o.numpy()) for o in s.out}
    return s


def _download_async(s, grids, out):
    for g, o in zip(grids, out):
        if s.lib.grhd2_gpu_download_async(g._h, s.ptr[id(o)], None):
            raise RuntimeError("download failed")


def run(state):
    s, c = state, state.case
    call = c["call"]
    if call == "step":
        g = s.grids[0]
        g.upload(up=s.up0)
        g.cons_to_prim()
        g.step(s.dt)
        return g.download(want_p=False)[0]
    if call == "solve":
        g = s.grids[0]
        g.upload(p=s.p0)
        g.prim_to_cons()
        g.run(0.0, 1e30, c["steps"])
        return g.download(want_p=False)[0]
    if call == "rhs":
        g = s.grids[0]
        g.upload(p=s.p0)
        rhs = g.calc_rhs()
        return rhs if c["precision"] == "fp64" else rhs.astype(np.float32)  # FP32 arithmetic, widened by the library
    if call == "run":
        s.grids[0].run(0.0, 1e30, c["steps"])
        _download_async(s, s.grids, s.out)
        return s.out
    for b, grids, out in s.subs:
        if call == "e2e":
            for g, o in zip(grids, out):
                if s.lib.grhd2_gpu_upload_async(g._h, s.ptr[id(o)], None):
                    raise RuntimeError("upload failed")
            b.cons_to_prim()
        b.step(c["steps"], graph=True)
        _download_async(s, grids, out)
    return s.out


def work(case):
    """Bytes: five primitives, u and up read, up and the primitives written by each of the
    three stages of a step (the right-hand side alone: primitives read, rhs written), and
    the state's copies out and in.  Operations: an ENO-type reconstruction of five variables
    on both sides of each face (90 each), the Riemann flux (250), sources (350 off flat
    space), con2prim (200) and the stage combination (30)."""
    if case["call"] == "serve":
        reqs = make_stream(n=case["grids"], seed=case["stream"])
        sizes = [(r.cells, 1, r.kind == "michel") for r in reqs]
    else:
        dirs = 1 + (case["ny"] > 1) + (case["nz"] > 1)
        curved = case["problem"] not in ("sod", "kelvin_helmholtz")
        sizes = [(case["nx"] * case["ny"] * case["nz"], dirs, curved)] * case["grids"]
    n = sum(z for z, _, _ in sizes)
    rhs = sum(z * (d * 1150 + (350 if curved else 0)) for z, d, curved in sizes)
    if case["call"] == "rhs":
        return {"bytes": 80 * n, "flops": rhs}
    el = 8 if case["precision"] == "fp64" else 4
    carry = 80 if case["precision"] == "mixed_comp64" else 0  # the compensated state: u's carry read, up's read and written
    copies = {"step": 2, "solve": 2, "e2e": 2}.get(case["call"], 1)
    return {"bytes": n * (case["steps"] * 3 * (2 * 5 * el + 3 * 40 + carry) + copies * 40),
            "flops": case["steps"] * 3 * (rhs + 230 * n)}


# ---- the path in plain 64-bit torch ----------------------------------------------------------
def exact(case, seed):
    dev = "cuda" if torch.cuda.is_available() and case["call"] != "serve" else "cpu"
    out = []
    pbs = _problems(case, seed)
    order = [q for k in range(4) for q in range(k, len(pbs), 4)] if case["call"] == "e2e" and len(pbs) >= 4 else None
    if case["call"] == "e2e" and len(pbs) < 4:
        order = list(range(len(pbs)))
    for pb in (pbs if order is None else [pbs[q] for q in order]):
        out.append(_Path(pb, _initial(pb), dev).advance(case).cpu().numpy())
    return out[0] if case["call"] in ("step", "solve", "rhs") else out


def _tensor(ptr, shape, dev):
    return torch.from_numpy(np.ctypeslib.as_array(ptr, shape=shape).copy()).to(dev)


class _Path:
    """One grid: state q (5, nz, ny, nx); tables per (ny, nx) cell and per face, no ghosts."""

    def __init__(self, pb, p0, dev):
        self.pb, self.dev, self.c = pb, dev, pb.config(0)
        self.nx, self.ny, self.nz, g = pb.nx, pb.ny, pb.nz, pb.ng
        nx, ny = self.nx, self.ny
        m = pb.metric_view()
        self.alpha = _tensor(m.alpha_c, (ny, nx), dev)
        self.beta = _tensor(m.beta_c, (ny, nx, 3), dev)
        self.gam = _tensor(m.gamma_c, (ny, nx, 3, 3), dev)
        self.gin = _tensor(m.gamma_inv_c, (ny, nx, 3, 3), dev)
        self.sqg = _tensor(m.sqrt_gamma_c, (ny, nx), dev)
        self.gmn = _tensor(m.gmunu_c, (ny, nx, 4, 4), dev)
        self.ch0 = _tensor(m.chris_c, (ny, nx, 4, 4, 4), dev)[..., 0]
        self.dg = _tensor(m.dg_c, (ny, nx, 3, 4, 4), dev)
        self.dlna = _tensor(m.dlna_c, (ny, nx, 4), dev)
        self.faces = {}
        for d, s, n in ((1, "x", (ny, nx + 1)), (2, "y", (ny + 1, nx)), (3, "z", (ny, nx))):
            if (self.nx, self.ny, self.nz)[d - 1] > 1:
                self.faces[d] = [_tensor(getattr(m, f"{f}_f_{s}"), n + t, dev) for f, t in
                                 (("alpha", ()), ("beta", (3,)), ("gamma", (3, 3)), ("sqrt_gamma", ()))]
        self.zero = None
        if ny > 1 and self.c.geom_kind >= 2:
            yf = np.ctypeslib.as_array(m.y_face, shape=(ny + 1,))
            self.zero = torch.from_numpy(np.abs(np.sin(yf)) <= 64 * np.finfo(float).eps).to(dev)
        self.case_id = self.c.case_id
        if self.case_id == 7:
            b = pb.bc_view()
            self.inj = _tensor(b.michel_injector, (pb.nz, ny, g, 5), dev).permute(3, 0, 1, 2)
        inner = p0[g + 1:g + 1 + pb.nz, g + 1:g + 1 + ny, g + 1:g + 1 + nx, :]
        self.q = torch.from_numpy(np.ascontiguousarray(inner.transpose(3, 0, 1, 2))).to(dev)
        self.minkowski = self.c.metric_kind == 0
        self.srhd = self.minkowski and self.c.geom_kind == 0

    # -- boundaries: three ghost layers along direction d (1, 2, 3) -------------------------
    def pad(self, d):
        q, cs, ax = self.q, self.case_id, 4 - d
        n = q.shape[ax]
        idx = torch.arange(-2, n + 4, device=self.dev)  # cells -2 .. n+3
        if d == 1 and cs not in (4, 6):
            src = idx.clamp(1, n)
        elif d == 2 and cs in (11, 12):
            src = torch.where(idx < 1, 1 - idx, torch.where(idx > n, 2 * n + 1 - idx, idx))
        else:
            src = (idx - 1) % n + 1
        e = q.index_select(ax, src - 1).clone()
        if d == 1 and cs == 7:
            g = self.inj.shape[-1]
            e[..., n + 3:n + 3 + g] = self.inj
        elif d == 1 and cs >= 9:
            va = self.beta[:, :, 0] / self.alpha
            for sl, col, lo in ((slice(0, 3), 0, True), (slice(n + 3, n + 6), n - 1, False)):
                thin = e[0, ..., sl] < 1e-6
                e[0, ..., sl] = e[0, ..., sl].clamp(min=self.c.rho_floor)
                e[1, ..., sl] = e[1, ..., sl].clamp(min=self.c.p_floor)
                f = torch.minimum if lo else torch.maximum
                e[2, ..., sl] = f(e[2, ..., sl], va[:, col][None, :, None].expand_as(e[2, ..., sl]))
                if lo and cs in (9, 10):
                    for v in (3, 4):
                        e[v, ..., sl] = torch.where(thin, torch.zeros_like(e[v, ..., sl]), e[v, ..., sl])
        elif d == 2 and cs in (11, 12):
            ghost = torch.cat([torch.arange(3), torch.arange(n + 3, n + 6)]).to(self.dev)
            part = e.index_select(ax, ghost)
            if cs == 12:
                part = part.roll(q.shape[1] // 2, dims=1)
            part[3] = -part[3]
            e.index_copy_(ax, ghost, part)
        return e.movedim(ax, 0)  # stencil index first

    # -- reconstruction --------------------------------------------------------------------
    def interface(self, d):
        e, n = self.pad(d), (self.nx, self.ny, self.nz)[d - 1]
        s = [e[m:m + n + 1] for m in range(6)]  # face i: cells i-2 .. i+3
        rec = self.c.rec_method
        left, right = s[:5], s[:0:-1]
        curved_x = not self.minkowski and d == 1
        face = torch.arange(n + 1, device=self.dev)
        shape = (n + 1,) + (1,) * (s[0].dim() - 2)
        godunov = ((face <= 0) & torch.tensor(curved_x, device=self.dev)).reshape(shape)
        shock = smooth = torch.zeros_like(godunov)
        if self.c.shock_sensor:
            jump = []
            for v, fl in ((1, self.c.p_floor), (0, self.c.rho_floor)):
                w = torch.stack([x[:, v] for x in s[:5]])
                hi, lo = w.amax(0), w.amin(0)
                jump.append(torch.where(hi > 1e3 * fl, (hi - lo) / lo.clamp(min=fl), torch.zeros_like(hi)))
            pj, rj = jump
            atm = 1e2 * self.c.rho_floor
            godunov = godunov | (s[2][:, 0] <= atm) | (s[3][:, 0] <= atm) | (pj >= 10) | (rj >= 10)
            shock = (pj >= 0.8) | (rj >= 0.5)
            smooth = (pj >= 0.4) | (rj >= 0.15)
            if rec == 4 and not self.minkowski:
                near = torch.zeros_like(face, dtype=torch.bool)
                if d == 1:
                    near = face <= 3
                if d == 2:
                    near = (face <= 2) | (face >= n - 2)
                smooth = smooth | near.reshape(shape)
        out = []
        for w in (left, right):
            if rec == 2:
                r = w[2] + 0.5 * _slope(w[2] - w[1], w[3] - w[2], self.c.tvd_limiter)
            elif rec == 3:
                r = _weno3(w[1], w[2], w[3])
            elif rec == 4:
                r = _mp5(*w[:5])
            else:
                r = _weno5(*w[:5])
            if self.c.shock_sensor:
                r = torch.where(smooth.unsqueeze(1), _weno3(w[1], w[2], w[3]), r)
                mc = w[2] + 0.5 * _slope(w[2] - w[1], w[3] - w[2], 3)
                r = torch.where(shock.unsqueeze(1), mc, r)
            if rec == 2 and not self.c.shock_sensor:
                godunov = torch.zeros_like(godunov)
            r = torch.where(godunov.unsqueeze(1), w[2], r).movedim(1, 0).clone()
            r[0] = r[0].clamp(min=self.c.rho_floor)
            r[1] = r[1].clamp(min=self.c.p_floor)
            out.append(r.movedim(1, 4 - d))  # (5, nz, ny, nx) with faces along d
        return out

    # -- Riemann solvers -------------------------------------------------------------------
    def cap(self, q, g):
        v = q[2:5]
        v2 = sum(g[..., a, b] * v[a] * v[b] for a in range(3) for b in range(3))
        over = v2 >= self.c.v_max
        f = torch.where(over, (self.c.v_max / v2.clamp(min=1e-300)).sqrt(), torch.ones_like(v2))
        return v * f, torch.where(over, torch.full_like(v2, self.c.v_max), v2)

    def flux_and_cons(self, q, d, al, be, g, sq):
        v, v2 = self.cap(q, g)
        vc = [sum(g[..., a, b] * v[b] for b in range(3)) for a in range(3)]
        h = 1 + self.c.g1 * q[1] / q[0]
        W = 1 / (1 - v2).sqrt()
        ve = al * v[d - 1] - be
        r = q[0] * h * W * W
        D = q[0] * W
        f = [D * ve, r * ve + q[1] * be - D * ve] + [r * vc[a] * ve + (al * q[1] if a == d - 1 else 0) for a in range(3)]
        u = [D, r - q[1] - D] + [r * vc[a] for a in range(3)]
        return torch.stack(f) * sq, torch.stack(u) * sq

    def speeds(self, q, d, al, be, g, gup):
        v, v2 = self.cap(q, g)
        h = 1 + self.c.g1 * q[1] / q[0]
        c2 = self.c.adb_idx * q[1] / (q[0] * h)
        vn = v[d - 1]
        t = al / (1 - v2 * c2)
        rad = (1 - v2) * (gup * (1 - v2 * c2) - vn * vn * (1 - c2))
        t2 = c2.sqrt() * rad.clamp(min=0).sqrt()
        e = torch.stack([al * vn - be, t * (vn * (1 - c2) + t2) - be, t * (vn * (1 - c2) - t2) - be, torch.zeros_like(vn)])
        return e.amin(0), e.amax(0)

    def hlle(self, qL, qR, d, al, be, g, sq, gup):
        fL, uL = self.flux_and_cons(qL, d, al, be, g, sq)
        fR, uR = self.flux_and_cons(qR, d, al, be, g, sq)
        a, b = self.speeds(qL, d, al, be, g, gup), self.speeds(qR, d, al, be, g, gup)
        am, ap = torch.minimum(a[0], b[0]), torch.maximum(a[1], b[1])
        f = (ap * fL - am * fR + ap * am * (uR - uL)) / (ap - am)
        return torch.where((ap - am).abs() < 1e-14, torch.zeros_like(f), f)

    def hllc(self, qL, qR, d, al, be, g, sq, gup, gi):
        cof = _coframe(g, gi, d)
        ok = torch.ones_like(al + qL[0], dtype=torch.bool)
        loc, tiny = [], 2.3e-308
        for q in (qL, qR):
            v = torch.stack([sum(cof[..., a, i] * q[2 + i] for i in range(3)) for a in range(3)])
            v2 = (v * v).sum(0)
            h = 1 + self.c.g1 * q[1] / q[0]
            c2 = self.c.adb_idx * q[1] / (q[0] * h)
            ok = ok & (v2 < self.c.v_max) & (c2 < 1) & (q[0] > 0)
            v2s = v2.clamp(max=self.c.v_max)
            W = 1 / (1 - v2s).sqrt()
            D, r = q[0] * W, q[0] * h * W * W
            u = torch.stack([D, r - q[1] - D, r * v[0], r * v[1], r * v[2]])
            f = torch.stack([D * v[0], u[2] - D * v[0], u[2] * v[0] + q[1], u[3] * v[0], u[4] * v[0]])
            den = 1 - v2s * c2
            rad = (1 - v2s) * (den - v[0] ** 2 * (1 - c2))
            ac = c2.sqrt() * rad.clamp(min=0).sqrt()
            ok = ok & (den > 1e-14) & (rad >= -1e-12)
            loc.append((u, f, (v[0] * (1 - c2) - ac) / den, (v[0] * (1 - c2) + ac) / den, v[0], q[1]))
        (uL, fL, l0, l1, vL, pL), (uR, fR, r0, r1, vR, pR) = loc
        ll, lr = torch.minimum(l0, r0), torch.maximum(l1, r1)
        w = be / (al * gup.sqrt()) + torch.zeros_like(ll)
        ok = ok & (lr - ll > 1e-13)
        uh = (lr * uR - ll * uL + fL - fR) / (lr - ll)
        fh = (lr * fL - ll * fR + lr * ll * (uR - uL)) / (lr - ll)
        A, B, C = fh[1] + fh[0], -(uh[1] + uh[0] + fh[2]), uh[2]
        disc = B * B - 4 * A * C
        scale = torch.maximum(B * B, (4 * A * C).abs()).clamp(min=tiny)
        star = ok & (disc >= -1e-12 * scale)
        sd = disc.clamp(min=0).sqrt()
        quad = A.abs() > 1e-13 * torch.maximum(B.abs(), C.abs()).clamp(min=tiny)
        big = torch.maximum(B.abs(), sd).clamp(min=tiny)
        root = torch.where((-B - sd).abs() > 1e-14 * big, (-B - sd) / (2 * A), 2 * C / (-B + sd))
        ls = torch.where(quad, root, -C / B)
        tol = 1e-10 * torch.maximum(ll.abs(), lr.abs()).clamp(min=1)

        def valid(x):
            return torch.isfinite(x) & (x >= ll - tol) & (x <= lr + tol) & (x.abs() <= 1 + tol)

        alt = (-B + sd) / (2 * A)
        ls = torch.where(~valid(ls) & quad & valid(alt), alt, ls)
        star = star & valid(ls)
        ls = torch.minimum(lr, torch.maximum(ll, ls))
        ps = []
        for lam, u, v, p in ((ll, uL, vL, pL), (lr, uR, vR, pR)):
            den = 1 - lam * ls
            star = star & (den.abs() > 1e-13) & ((lam - ls).abs() > 1e-13)
            ps.append(((lam * (u[1] + u[0]) - u[2]) * ls - (u[2] * (lam - v) - p)) / den)
        big = torch.stack([(uL[1] + uL[0]).abs(), (uR[1] + uR[0]).abs(), uL[2].abs(), uR[2].abs()]).amax(0).clamp(min=tiny)
        ptol = 1e-8 * torch.stack([pL.abs(), pR.abs(), ps[0].abs(), ps[1].abs()]).amax(0).clamp(min=tiny) + 1e2 * 2.220446049250313e-16 * big
        star = star & ((ps[0] - ps[1]).abs() <= ptol)
        pst = 0.5 * (ps[0] + ps[1])
        side = []
        zero, one = torch.zeros_like(ls), torch.ones_like(ls)
        push = torch.stack([zero, ls, one, zero, zero])
        for lam, u, f in ((ll, uL, fL), (lr, uR, fR)):
            us = (lam * u - f + pst * push) / (lam - ls)
            E, m2 = us[1] + us[0], (us[2:] ** 2).sum(0)
            sc = torch.maximum(E * E, us[0] ** 2 + m2).clamp(min=tiny)
            star = star & (us[0] > 0) & (E > 0) & (E * E - us[0] ** 2 - m2 > 1e-13 * sc) & torch.isfinite(us).all(0)
            side.append((us, f + lam * (us - u)))
        pick = [torch.where(w <= ls, a, b) for a, b in zip(*side)]
        us = torch.where(w <= ll, uL, torch.where(w >= lr, uR, pick[0]))
        fs = torch.where(w <= ll, fL, torch.where(w >= lr, fR, pick[1]))
        use = ok & (star | (w <= ll) | (w >= lr))
        mf = (fs - w * us) * (sq * al * gup.sqrt())
        flux = torch.stack([mf[0], mf[1]] + [sum(cof[..., a, i] * mf[2 + a] for a in range(3)) for i in range(3)])
        return torch.where(use, flux, self.hlle(qL, qR, d, al, be, g, sq, gup))

    # -- right-hand side, con2prim, stages ---------------------------------------------------
    def rhs(self):
        out = self.sources()
        for d in self.faces:
            al, be, g, sq = self.faces[d]
            det = _det(g)
            gi = _inverse(g, det)
            args = (al, be[..., d - 1], g, sq, gi[..., d - 1, d - 1])
            qL, qR = self.interface(d)
            f = self.hllc(qL, qR, d, *args, gi) if self.c.riemann == 2 else self.hlle(qL, qR, d, *args)
            if d == 2 and self.zero is not None:
                f = torch.where(self.zero[:, None], torch.zeros_like(f), f)
            ax, n = 4 - d, (self.nx, self.ny, self.nz)[d - 1]
            out = out - (f.narrow(ax, 1, n) - f.narrow(ax, 0, n)) / (self.c.dx, self.c.dy, self.c.dz)[d - 1]
        return out

    def sources(self):
        q = self.q
        if self.srhd:
            return torch.zeros_like(q)
        v, v2 = self.cap(q, self.gam)
        h = 1 + self.c.g1 * q[1] / q[0]
        W = 1 / (1 - v2).sqrt()
        u = [W / self.alpha] + [W * (v[a] - self.beta[..., a] / self.alpha) for a in range(3)]
        T = {(m, n): q[0] * h * u[m] * u[n] + q[1] * self.gmn[..., n, m] for m in range(4) for n in range(m, 4)}
        at = lambda m, n: T[(m, n) if m <= n else (n, m)]  # noqa: E731
        pairs = [(m, n) for m in range(4) for n in range(4)]
        s = [sum(0.5 * at(m, n) * self.dg[..., d, n, m] for m, n in pairs) for d in range(3)]
        e = sum(at(m, 0) * self.dlna[..., m] for m in range(4)) - sum(at(m, n) * self.ch0[..., n, m] for m, n in pairs)
        f = self.alpha * self.sqg
        return torch.stack([torch.zeros_like(e), e * f * self.alpha] + [x * f for x in s])

    def prim_to_cons(self):
        zero = torch.zeros_like(self.alpha)
        return self.flux_and_cons(self.q, 1, zero, zero, self.gam, self.sqg)[1]

    def cons_to_prim(self, cs):
        rho_fl, p_fl, g1, gi, sq = self.c.rho_floor, self.c.p_floor, self.c.g1, self.gin, self.sqg
        dfl = rho_fl * sq + torch.zeros_like(cs[0])
        tfl = p_fl * (g1 - 1) * sq + torch.zeros_like(cs[0])
        floor = cs[0] <= dfl
        D, tau, S = cs[0], cs[1], cs[2:5]

        def sq2(S):
            return sum(gi[..., a, b] * S[a] * S[b] for a in range(3) for b in range(3))

        smax = ((tau + D) ** 2 - D * D).clamp(min=0) * self.c.v_max
        s2 = sq2(S)
        S = S * torch.where((s2 > smax) & (s2 > 1e-20) & ~floor, (smax / s2.clamp(min=1e-300)).sqrt(), torch.ones_like(s2))
        Q2 = sq2(S)
        hi = torch.maximum(2 * (Q2.clamp(min=0).sqrt() + D) / D.clamp(min=rho_fl), torch.full_like(D, 1e3))

        def value(W):
            den = g1 * W * W - 1
            V = (g1 * W * W * (tau + D) - D * W) / den
            return V, V * V * (1 - 1 / (W * W)) - Q2, (g1 * W * (D * W - 2 * (tau + D)) + D) / (den * den)

        W, top = torch.ones_like(D), value(hi)[1]
        x0, x1 = W, hi
        for _ in range(45):  # log-spaced bisection, then Newton from a bracketed start
            mid = (x0 * x1).sqrt()
            up = value(mid)[1] > 0
            x0, x1 = torch.where(up, x0, mid), torch.where(up, mid, x1)
        W = 0.5 * (x0 + x1)
        for _ in range(3):
            V, f, dV = value(W)
            W3 = W * W * W
            step = f * W3 / (2 * V * (dV * (W3 - W) + V))
            W = torch.where(torch.isfinite(step), torch.minimum(x1, torch.maximum(x0, W - step)), W)
        W = torch.where(Q2 < 1e-14, torch.ones_like(W), torch.where(top.abs() < 1e-14, hi, W))
        floor = floor | ((top < 0) & (Q2 >= 1e-14) & (top.abs() >= 1e-14))
        V = value(W)[0]
        floor = floor | ~(V > 0)
        pr = torch.stack([D / (W * sq), (V - tau - D) / sq] + [sum(gi[..., a, b] * S[b] for b in range(3)) / V for a in range(3)])
        v2 = sum(self.gam[..., a, b] * pr[2 + a] * pr[2 + b] for a in range(3) for b in range(3))
        floor = floor | ~((pr[0] >= rho_fl) & (pr[1] >= p_fl) & (v2 < self.c.v_max))
        zero = torch.zeros_like(D)
        rest = torch.stack([zero + rho_fl, zero + p_fl, zero, zero, zero])
        still = torch.stack([dfl, tfl, zero, zero, zero])
        self.q = torch.where(floor, rest, pr)
        return torch.where(floor, still, torch.cat([cs[:2], S]))

    def dt(self):
        inv = 0.0
        for d, dx in zip(self.faces, [x for x, n in zip((self.c.dx, self.c.dy, self.c.dz), (self.nx, self.ny, self.nz)) if n > 1]):
            inv += float((self.alpha * self.gin[..., d - 1, d - 1].sqrt() + self.beta[..., d - 1].abs()).max()) / dx
        return self.c.cfl / inv

    def advance(self, case):
        if case["call"] == "rhs":
            out = self.rhs()
        else:
            out = self.prim_to_cons()
            dt = self.dt()
            if case["call"] in ("step", "e2e"):
                out = self.cons_to_prim(out)
            for _ in range(case["steps"]):
                u = out
                out = self.cons_to_prim(u + self.rhs() * dt)
                out = self.cons_to_prim(0.75 * u + 0.25 * (out + self.rhs() * dt))
                out = self.cons_to_prim((u + 2 * (out + self.rhs() * dt)) / 3)
        return out.permute(1, 2, 3, 0).contiguous()


def _det(g):
    return (g[..., 0, 0] * (g[..., 1, 1] * g[..., 2, 2] - g[..., 1, 2] ** 2)
            - g[..., 0, 1] * (g[..., 0, 1] * g[..., 2, 2] - g[..., 1, 2] * g[..., 0, 2])
            + g[..., 0, 2] * (g[..., 0, 1] * g[..., 1, 2] - g[..., 1, 1] * g[..., 0, 2]))


def _inverse(g, det):
    cof = lambda a, b: (g[..., (b + 1) % 3, (a + 1) % 3] * g[..., (b + 2) % 3, (a + 2) % 3]  # noqa: E731
                        - g[..., (b + 1) % 3, (a + 2) % 3] * g[..., (b + 2) % 3, (a + 1) % 3])
    return torch.stack([torch.stack([cof(a, b) / det for b in range(3)], -1) for a in range(3)], -2)


def _coframe(g, gi, d):
    """Covectors of the orthonormal frame whose first leg is normal to the faces of direction d."""
    dot = lambda x, y: (g * x[..., :, None] * y[..., None, :]).sum((-1, -2))  # noqa: E731
    legs = [gi[..., d - 1] / gi[..., d - 1, d - 1, None].sqrt()]
    for t in ((1, 2), (2, 0), (0, 1))[d - 1]:
        s = torch.zeros_like(legs[0])
        s[..., t] = 1
        for e in legs:
            s = s - dot(s, e)[..., None] * e
        legs.append(s / dot(s, s)[..., None].sqrt())
    return torch.stack([(g * e[..., None, :]).sum(-1) for e in legs], -2)


def _minmod(a, b):
    return 0.5 * (a.sign() + b.sign()) * torch.minimum(a.abs(), b.abs())


def _slope(a, b, lim):
    s = a.sign()
    if lim == 2:
        sl = s * torch.maximum(torch.minimum(2 * a.abs(), b.abs()), torch.minimum(a.abs(), 2 * b.abs()))
        return torch.where(a * b <= 0, torch.zeros_like(a), sl)
    if lim == 3:
        x, y, z = 2 * b, 0.5 * (a + b), 2 * a
        s = x.sign()
        return s * torch.minimum(torch.minimum(x.abs(), s * y), s * z).clamp(min=0)
    return _minmod(a, b)


def _weno3(qm, q0, qp):
    b0, b1 = (q0 - qp) ** 2, (qm - q0) ** 2
    sensor = (b0 - b1).abs() / (torch.maximum(b0, b1) + 1e-14)
    eh = 1e-14 + (qm * qm + q0 * q0 + qp * qp) * torch.exp(-10 * sensor)
    a0, a1 = (2 / 3) / (eh + b0) ** 2, (1 / 3) / (eh + b1) ** 2
    return (a0 * (0.5 * q0 + 0.5 * qp) + a1 * (-0.5 * qm + 1.5 * q0)) / (a0 + a1)


def _weno5(a, b, c, d, e):
    b0 = 13 / 12 * (c - 2 * d + e) ** 2 + 0.25 * (3 * c - 4 * d + e) ** 2
    b1 = 13 / 12 * (b - 2 * c + d) ** 2 + 0.25 * (b - d) ** 2
    b2 = 13 / 12 * (a - 2 * b + c) ** 2 + 0.25 * (a - 4 * b + 3 * c) ** 2
    tau = (b0 - b2).abs()
    a0, a1, a2 = (w * (1 + tau / (1e-14 + x)) for w, x in ((0.3, b0), (0.6, b1), (0.1, b2)))
    p0, p1, p2 = c / 3 + 5 / 6 * d - e / 6, -b / 6 + 5 / 6 * c + d / 3, a / 3 - 7 / 6 * b + 11 / 6 * c
    return (a0 * p0 + a1 * p1 + a2 * p2) / (a0 + a1 + a2)


def _mp5(a, b, c, d, e):
    low = (2 * a - 13 * b + 47 * c + 27 * d - 3 * e) / 60
    mp = c + _minmod(d - c, 4 * (c - b))
    dm, d0, dp = a - 2 * b + c, b - 2 * c + d, c - 2 * d + e

    def minmod4(w, x, y, z):
        s = 0.125 * (w.sign() + x.sign()) * ((w.sign() + y.sign()) * (w.sign() + z.sign())).abs()
        return s * torch.stack([w.abs(), x.abs(), y.abs(), z.abs()]).amin(0)

    jp, jm = minmod4(4 * d0 - dp, 4 * dp - d0, d0, dp), minmod4(4 * d0 - dm, 4 * dm - d0, d0, dm)
    ul, md, lc = c + 4 * (c - b), 0.5 * (c + d) - 0.5 * jp, c + 0.5 * (c - b) + 4 / 3 * jm
    lo = torch.maximum(torch.minimum(torch.minimum(c, d), md), torch.minimum(torch.minimum(c, ul), lc))
    hi = torch.minimum(torch.maximum(torch.maximum(c, d), md), torch.maximum(torch.maximum(c, ul), lc))
    return torch.where((low - c) * (low - mp) < 1e-10, low, low + _minmod(lo - low, hi - low))
