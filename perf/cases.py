"""The calls this framework is used for, over the sizes it is used at.

A case is one stretch of a run between two looks at it: the simulation (or the
pool of simulations) advances a number of steps and the fields its user wants
then are read back.  A domain's user reads the five fields of a movie frame
(bed, depth, speed, concentration, deposited mass); a pool's user reads depth
and concentration of every scenario, as the request loop does.

Most cases start in the middle of an event: bed, Ks and a snapshot of sheet
flow with suspended and deposited sediment, with the distributions that a run
has after some minutes of rain (depths around 1 mm, speeds of centimetres per
second, fine classes suspended and coarse ones mostly deposited).  One starts
from the dry bed, as every run does, and so does the example of the reference.
Rain never ends and the end time is far off, so that many passes can follow one
another.
"""
import math

import numpy as np
import torch

from swehr_b200 import workloads as W
from swehr_b200.lib import Pool, Simulation
from swehr_b200.params import FIELD_NAMES, FP64, MIXED, REFERENCE_DEFAULTS

FRAME = ("z", "h", "vel", "totsed", "totm")
RESULT = ("h", "totsed")
FORMS = {"fp64": FP64, "mixed": MIXED}


def _domain(**kw):
    case = dict(kind="domain", terrain="fractal", nx=64, ny=64, dx=1.0, classes=7, form="fp64", wet=True, ks=True,
                storm=False, solid=False, inflow=False, budget=False, walls="0111", steps=100)
    case.update(kw)
    return case


def _pool(**kw):
    case = dict(kind="pool", count=16, side_min=64, side_max=1024, classes_min=7, classes_max=7, form="mixed",
                chunk=32, chunks=1)
    case.update(kw)
    return case


def listed():
    return [
        # the reference's own example, 3 x 51 cells with the sediment-laden inflow, from the dry bed
        _domain(name="example_fp64", terrain="plane", nx=3, ny=51, dx=0.25, classes=1, wet=False, ks=False,
                inflow=True, walls="1011", steps=128),
        # the 200 x 50 hillslope, the size most single catchments have, in both forms; the mixed one with its budget
        _domain(name="hillslope_fp64", terrain="hillslope", nx=200, ny=50, ks=False, steps=128),
        _domain(name="hillslope_mixed_budget", terrain="hillslope", nx=200, ny=50, ks=False, form="mixed",
                budget=True, steps=128),
        # a town: ragged sizes, ten classes, buildings as interior solid cells
        _domain(name="town_fp64", nx=517, ny=389, classes=10, solid=True),
        # the first steps of a storm on a dry catchment: most cells see no water
        _domain(name="dry_start_fp64", nx=1024, ny=1024, dx=2.0, wet=False, storm=True),
        # an odd-sized catchment with a class count that has no kernel of its own
        _domain(name="odd_mixed", nx=1023, ny=1531, classes=5, form="mixed"),
        # the roofline domain in both forms
        _domain(name="large_fp64", nx=4096, ny=4096, dx=2.0, steps=60),
        _domain(name="large_mixed", nx=4096, ny=4096, dx=2.0, form="mixed"),
        # a moving storm with ten classes: water and sediment along its track, film or dry bed elsewhere
        _domain(name="storm_mixed", nx=2048, ny=2048, classes=10, form="mixed", storm=True),
        # ensembles of catchments of many sizes, stepped together in both forms
        _pool(name="ensemble_fp64", form="fp64", chunks=2),
        _pool(name="ensemble_mixed", chunks=3),
        # a serving mix: requests of 5 to 10 classes, advanced in the chunks of the request loop
        _pool(name="serving_mixed", count=24, side_min=32, classes_min=5, classes_max=10, chunk=16, chunks=4),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    form = rng.choice(["fp64", "mixed"])
    if rng.random() < 0.25:
        lo = _log_int(rng, 16, 128)
        s_lo = rng.randint(1, 10)
        return _pool(count=rng.randint(2, 24), side_min=lo, side_max=_log_int(rng, 2 * lo, 1024), classes_min=s_lo,
                     classes_max=rng.choice([s_lo, min(16, s_lo + rng.randint(1, 6))]), form=form,
                     chunk=rng.randint(8, 48), chunks=rng.randint(1, 3))
    storm = rng.random() < 0.2
    return _domain(terrain=rng.choice(["fractal", "fractal", "hillslope"]), nx=_log_int(rng, 3, 2500),
                   ny=_log_int(rng, 3, 2500), dx=rng.choice([0.5, 1.0, 2.0]),
                   classes=rng.choice([1, 2, 3, 4, 5, 6, 7, 7, 7, 8, 10, 10, 12, 16]), form=form,
                   wet=rng.random() < 0.75, ks=rng.random() < 0.6, storm=storm, solid=rng.random() < 0.15,
                   budget=rng.random() < 0.15, walls=rng.choice(["0111", "0111", "0000", "1011", "0101"]),
                   steps=rng.randint(32, 128))


# ------------------------------------------------------------------ inputs
def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _fractal(nx, ny, relief, dev, gen):
    """A power-law surface (Hurst 0.8) of the given relief."""
    kx = torch.fft.fftfreq(nx, device=dev, dtype=torch.float64)[:, None]
    ky = torch.fft.rfftfreq(ny, device=dev, dtype=torch.float64)[None, :]
    k2 = kx * kx + ky * ky
    k2[0, 0] = 1.0
    amp = k2 ** -0.9
    amp[0, 0] = 0.0
    noise = torch.fft.rfft2(torch.randn(nx, ny, device=dev, dtype=torch.float64, generator=gen))
    z = torch.fft.irfft2(noise * amp, s=(nx, ny))
    z = z - z.min()
    return z * (relief / max(float(z.max()), 1e-300))


def _inputs(case, seed):
    """The case's parameters, input arrays and snapshot: (W.Case, {(field, class): array}), all from the seed."""
    dev = _device()
    gen = torch.Generator(device=dev)
    gen.manual_seed(int(seed))
    rng = np.random.default_rng(int(seed))
    nx, ny, S, dx = case["nx"], case["ny"], case["classes"], case["dx"]

    def normal():
        return torch.randn(nx, ny, device=dev, dtype=torch.float64, generator=gen)

    x = (torch.arange(nx, device=dev, dtype=torch.float64) * dx)[:, None]
    y = (torch.arange(ny, device=dev, dtype=torch.float64) * dx)[None, :]
    if case["terrain"] == "plane":            # the example's bed rises along j
        topo = 0.7002 * y + 0.0 * x + 1e-4 * normal()
    elif case["terrain"] == "hillslope":
        topo = 0.1 * x + 0.005 * normal()
    else:
        topo = 0.03 * x + _fractal(nx, ny, 40.0 * min(1.0, max(nx, ny) * dx / 4096.0), dev, gen)
    ds = 2e-6 * 1000.0 ** (np.arange(S) / max(S - 1, 1)) if S > 1 else np.array([2e-4])
    pf = rng.dirichlet([2.0] * S)
    params = dict(nx=nx, ny=ny, dx=dx, tend=1.0e9, sclass=S, bndry=tuple(int(b) for b in case["walls"]),
                  inflow=int(case["inflow"]))
    if case["inflow"]:
        params.update(F=0.004, manning0=1.0, a=0.0, ad=0.0, h0=0.00099, mtstar0=3.0, J=30.0, rnum=2, rint=60.0,
                      stageint=1.0)
        rain = np.zeros(2)
    else:
        params = W.common_soil(**dict(params, rnum=30, rint=60.0))
        rain = rng.uniform(20.0, 120.0, size=30) * W.MMH
    radius, track = max(nx, ny) * dx / 8, ny * dx / 3      # the storm domain's proportions
    if case["storm"]:
        params.update(storm_peak=200 * W.MMH, storm_radius=radius, storm_x0=nx * dx / 2, storm_y0=track,
                      storm_vx=0.0, storm_vy=2.0)
    ks = None
    if case["ks"]:
        ks = ((5 * W.MMH) * torch.exp(0.5 * normal())).cpu().numpy()
    solid = None
    if case["solid"]:
        solid = np.zeros((nx, ny), dtype=np.int32)
        for _ in range(max(1, nx * ny // 4000)):
            i, j = int(rng.integers(0, nx)), int(rng.integers(0, ny))
            solid[i:i + int(rng.integers(2, 14)), j:j + int(rng.integers(2, 14))] = 1
    made = W.Case("case", params, topo.cpu().numpy(), rain, ds, pf, ks=ks, solid=solid)
    if not case["wet"]:
        return made, {}
    # the snapshot: sheet flow down the slope, fine classes in suspension
    gx, gy = torch.zeros_like(topo), torch.zeros_like(topo)
    gx[1:-1] = (topo[2:] - topo[:-2]) / (2 * dx)
    gy[:, 1:-1] = (topo[:, 2:] - topo[:, :-2]) / (2 * dx)
    norm = torch.sqrt(gx * gx + gy * gy) + 1e-12
    h = 1.0e-3 * torch.exp(0.35 * normal()) + 1e-5
    speed = 0.045 * torch.exp(0.4 * normal())
    snap = {("h", 0): h, ("hu", 0): -h * speed * gx / norm, ("hv", 0): -h * speed * gy / norm,
            ("vinf", 0): 5.0e-3 * torch.exp(0.2 * normal())}
    rhos = REFERENCE_DEFAULTS["rhos"]
    susp, bed = torch.exp(0.25 * normal()), torch.exp(0.15 * normal())
    totsed, totm = torch.zeros_like(h), torch.zeros_like(h)
    for k in range(S):
        sed = float(min(70.0, 70.0 * (ds[k] / 8e-6) ** -1.3)) * float(pf[k]) * 7.0 * min(1.0, 7.0 / S)
        snap["U", k + 1] = h * sed * susp
        snap["M", k + 1] = (0.05 + 0.45 * float(pf[k])) * bed * (0.3 if ds[k] < 4e-6 else 1.0)
        totsed = totsed + sed * susp / rhos
        totm = totm + snap["M", k + 1]
    snap["totsed", 0] = totsed
    snap["totm", 0] = totm
    snap["dep", 0] = totm / rhos
    snap["maxvel", 0] = 1.1 * speed
    snap["maxdepth", 0] = 1.1 * h
    if case["storm"]:                         # outside the storm's track the rain has not come yet
        out = ((x - nx * dx / 2).abs() > 1.3 * radius) | (y > track + radius)
        for key, v in snap.items():
            fill = {"h": 1e-5, "vinf": 1e-4, "maxdepth": 1e-5}.get(key[0], 0.0)
            snap[key] = torch.where(out, torch.full_like(v, fill), v)
    if solid is not None:                     # no water in a solid cell
        dry = torch.from_numpy(solid != 0).to(dev)
        for key, v in snap.items():
            snap[key] = torch.where(dry, torch.zeros_like(v), v)
    return made, {key: v.cpu().numpy() for key, v in snap.items()}


def _scenarios(case, seed):
    """The domain cases that a pool case is made of (the same sizes for every seed)."""
    rng = np.random.default_rng(7)
    made = []
    for s in range(case["count"]):
        side = int(round(math.exp(rng.uniform(math.log(case["side_min"]), math.log(case["side_max"])))))
        S = int(rng.integers(case["classes_min"], case["classes_max"] + 1))
        made.append((_domain(terrain="hillslope" if s % 4 == 3 else "fractal", nx=side, ny=side, classes=S,
                             wet=s % 8 != 5, ks=False, steps=case["chunk"] * case["chunks"]), 1000 * int(seed) + s))
    return made


# ------------------------------------------------------------- the measured call
def prepare(case, seed):
    form = FORMS[case["form"]]
    if case["kind"] == "domain":
        made, snap = _inputs(case, seed)
        sim = Simulation(made, precision=form, budget=case["budget"])
        for (name, k), a in snap.items():
            sim.write_field(name, a, k)
        return {"case": case, "sim": sim}
    pool = Pool(precision=form, max_classes=case["classes_max"], max_scenarios=case["count"])
    members = []
    for sub, sub_seed in _scenarios(case, seed):
        made, snap = _inputs(sub, sub_seed)
        made.params["tend"] = 36000.0
        sc = pool.submit(made)
        for (name, k), a in snap.items():
            a = np.ascontiguousarray(a)
            status = pool.L.swehr_write_field(sc.ctx, FIELD_NAMES[name], k, a.ctypes.data)
            assert status == 0, pool.L.swehr_last_error().decode()
        members.append(sc)
    return {"case": case, "pool": pool, "members": members}


def run(state):
    case = state["case"]
    if case["kind"] == "domain":
        sim = state["sim"]
        sim.advance(max_steps=case["steps"])
        out = sim.fields(FRAME)
        if case["budget"]:
            b = sim.budget()
            out["budget"] = np.array([b.rain_in, b.infiltration, b.outflow, b.water_now]
                                     + [b.sed_now[k] for k in range(case["classes"])])
        return out
    for _ in range(case["chunks"]):
        state["pool"].run(case["chunk"])
    return [sc.fields(RESULT) for sc in state["members"]]


# ------------------------------------------------------- bounds and comparison
def _work_domain(case, fields):
    cells, S, mixed = case["nx"] * case["ny"], case["classes"], case["form"] == "mixed"
    # a step reads and writes every prognostic field once and reads Ks
    per = 2 * (4 * (5 + S) + 8 * (2 + S)) + 4 * case["ks"] if mixed else 16 * (7 + 2 * S) + 8 * case["ks"]
    # the operations written out per cell, elementary functions counted as one
    return {"bytes": cells * (case["steps"] * per + fields * (8 + (4 if mixed else 8))),
            "flops": cells * case["steps"] * (320 + 55 * S)}


def work(case):
    if case["kind"] == "domain":
        return _work_domain(case, len(FRAME))
    parts = [_work_domain(dict(sub, form=case["form"]), len(RESULT)) for sub, _ in _scenarios(case, 0)]
    return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}


def tolerance(case):
    # Four times what the forms were seen to be off exact(): 3e-13 and 2e-6 in flow, and 5e-4 where film and dry bed
    # begin to flow (storms, dry starts): there the thresholds between film, shallow and deep water turn a last-bit
    # difference into a visible one in some cells.
    front = case["kind"] == "domain" and (case["storm"] or not case["wet"])
    if case["form"] == "fp64":
        return {"rel": 1e-9, "max": 1e-6}
    return {"rel": 2e-3, "max": 0.5} if front else {"rel": 2e-5, "max": 0.05}


# ------------------------------------------------------------ 64-bit restatement
class _Exact:
    """The step of SWEHR.c:808-1591 in float64 torch, one operation at a time."""

    def __init__(self, made, snap):
        dev = self.dev = _device()
        p = dict(REFERENCE_DEFAULTS)
        p.update(made.params)
        self.p, self.S = p, made.sclass
        t = lambda a: torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device=dev)  # noqa: E731
        self.ds, self.pf, self.rain = [float(v) for v in made.ds], [float(v) for v in made.pfrac], made.rain
        topo = np.array(made.topo, dtype=np.float64)
        self.solid = None
        if made.solid is not None:
            self._fill_solid(topo, made.solid)
            self.solid = torch.as_tensor(made.solid != 0, device=dev)
        self.z = t(topo)
        self.zp = self.z
        zero = torch.zeros_like(self.z)
        get = lambda name, k=0: t(snap[name, k]) if (name, k) in snap else zero.clone()  # noqa: E731
        self.h, self.hu, self.hv = get("h"), get("hu"), get("hv")
        self.vinf = get("vinf") if snap else zero + p["vinf0"]
        self.totm, self.dep, self.totsed = get("totm"), get("dep"), get("totsed")
        self.U = [get("U", k + 1) for k in range(self.S)]
        self.M = [get("M", k + 1) for k in range(self.S)]
        self.ks = zero + p["ks"] if made.ks is None else t(made.ks)
        self.t = 0.0
        self.sx0, self.sy0 = self._slope(self.z, 0), self._slope(self.z, 1)
        self.gz0 = p["g"] / torch.sqrt(self.sx0 ** 2 + self.sy0 ** 2 + 1)

    @staticmethod
    def _fill_solid(T, m):
        """Bed of solid cells from their neighbours, serially as initialcondition does (SWEHR.c:288-322)."""
        nx, ny = T.shape
        s = m != 0
        near = s.copy()
        near[1:] |= s[:-1]
        near[:-1] |= s[1:]
        near[:, 1:] |= s[:, :-1]
        near[:, :-1] |= s[:, 1:]
        for i, j in zip(*np.nonzero(near)):
            up, dn, ju, jd = min(i + 1, nx - 1), max(i - 1, 0), min(j + 1, ny - 1), max(j - 1, 0)
            if s[i, j]:
                for a, b in ((up, j), (dn, j), (up, ju), (up, jd), (dn, ju), (dn, jd), (i, ju), (i, jd)):
                    if not s[a, b]:
                        T[i, j] = T[a, b]
            else:
                for a, b in ((up, j), (dn, j), (i, ju), (i, jd)):
                    if s[a, b]:
                        T[a, b] = T[i, j]

    def _slope(self, z, dim):
        odx = 1 / self.p["dx"]
        z = z if dim == 0 else z.t()
        s = torch.empty_like(z)
        s[1:-1] = 0.5 * odx * (z[2:] - z[:-2])
        s[0] = odx * (z[1] - z[0])
        s[-1] = odx * (z[-1] - z[-2])
        return s if dim == 0 else s.t()

    def _hll(self, hl, hr, nl, nr, tl, tr, g, cl):
        film = self.p["hfilm"]
        cr = torch.sqrt(g * hr)
        d = nl + 2 * cl - nr - 2 * cr
        us = 0.5 * (nl + nr) + cl - cr
        cs = torch.sqrt(g * (d * d / (16 * g)))
        sl, sr, sm = torch.minimum(us - cs, nl - cl), torch.maximum(us + cs, nr + cr), us
        dl, dr = hl <= film, hr <= film
        sl = torch.where(dl, nr - 2 * cr, sl)
        sm = torch.where(dl, sl, sm)
        sr = torch.where(dl, nr + cr, sr)
        sl = torch.where(dr, nl - cl, sl)
        sr = torch.where(dr, nl + 2 * cl, sr)
        sm = torch.where(dr, sr, sm)
        pl, pr = hl * nl * nl + 0.5 * g * hl * hl, hr * nr * nr + 0.5 * g * hr * hr
        mid0 = (sr * (hl * nl) - sl * (hr * nr) + sl * sr * (hr - hl)) / (sr - sl)
        mid1 = (sr * pl - sl * pr + sl * sr * (hr * nr - hl * nl)) / (sr - sl)
        f0 = torch.where(sr <= 0, hr * nr, torch.where((sl <= 0) & (sr >= 0), mid0, hl * nl))
        f1 = torch.where(sr <= 0, pr, torch.where((sl <= 0) & (sr >= 0), mid1, pl))
        f2 = torch.where(sm >= 0, f0 * tl, f0 * tr)
        s = torch.maximum(torch.maximum(sl.abs(), sr.abs()), sm.abs())
        return f0, f1, f2, float(s.max())

    def _faces(self, dim, h, u, v, gz, sed, inflow):
        """Fluxes through the faces across `dim` (0: i, 1: j): three fluxes, the upwind concentrations and the
        largest wave speed; face f lies between cells f-1 and f, ghosts at both ends."""
        tr = (lambda a: a) if dim == 0 else (lambda a: a.t())
        h, n, t, gz = tr(h), tr(u if dim == 0 else v), tr(v if dim == 0 else u), tr(gz)
        sed = [tr(c) for c in sed]
        film = self.p["hfilm"]
        wall0, wall1 = self.p["bndry"][0 if dim == 0 else 1] == 1, self.p["bndry"][2 if dim == 0 else 3] == 1
        first = (h[:1], -n[:1] if wall0 else n[:1], t[:1])
        last = (h[-1:], -n[-1:] if wall1 else n[-1:], t[-1:])
        last_sed = [c[-1:] for c in sed]
        if inflow is not None:
            hin, hvin, sin = inflow
            full = torch.ones_like(h[-1:])
            last = (full * hin, full * (hvin / hin if hin > film else 0.0), full * 0.0)
            last_sed = [full * sin for _ in sed]
        hl, nl, tl = (torch.cat([a, b]) for a, b in zip(first, (h, n, t)))
        hr, nr, trt = (torch.cat([b, a]) for a, b in zip(last, (h, n, t)))
        g = torch.cat([gz[:1], gz])
        hr0, nr0, hl0, nl0, tl0, tr0 = hr, nr, hl, nl, tl, trt
        if self.solid is not None:
            s = tr(self.solid)
            none = torch.zeros_like(s[:1])
            sl, sr = torch.cat([none, s]), torch.cat([s, none])
            if dim == 0:
                sl[0], sr[-1], sl[-1] = False, False, False
                sr[0] = False
            else:                              # the test past the row reads the next row's first cell
                nxt = torch.zeros_like(s[:1])
                nxt[0, :-1] = self.solid[1:, 0]
                sr = torch.cat([s, nxt])
                sr[0] = False
            a, b = sl & ~sr, ~sl & sr
            hl, hr = torch.where(a, hr0, hl0), torch.where(b, hl0, hr0)
            nl = torch.where(a, torch.where(hr0 > film, -nr0, torch.zeros_like(nr0)), nl0)
            nr = torch.where(b, torch.where(hl0 > film, -nl0, torch.zeros_like(nl0)), nr0)
            tl, trt = torch.where(a, tr0, tl0), torch.where(b, tl0, tr0)
        f0, f1, f2, smax = self._hll(hl, hr, nl, nr, tl, trt, g, torch.sqrt(g * hl))
        up = f0 > 0
        cf = [torch.where(up, torch.cat([c[:1], c]), torch.cat([c, e])) for c, e in zip(sed, last_sed)]
        back = (lambda a: a) if dim == 0 else (lambda a: a.t())
        return back(f0), back(f1), back(f2), [back(c) for c in cf], smax

    def step(self):
        p, S = self.p, self.S
        film, g, rhos, rhow = p["hfilm"], p["g"], p["rhos"], p["rhow"]
        porod = rhos * (1 - p["phi"])
        h0, hu0, hv0, zc, zp = self.h, self.hu, self.hv, self.z, self.zp
        zero, one = torch.zeros_like(h0), torch.ones_like(h0)
        wet = h0 > film
        u, v = torch.where(wet, hu0 / h0, zero), torch.where(wet, hv0 / h0, zero)
        sed = []
        for k in range(S):
            c = torch.where(wet, self.U[k] / h0, zero)
            sed.append(torch.where(c < -1e-5, zero, c))
        sxp, syp = self._slope(zp, 0), self._slope(zp, 1)
        gzp = g / torch.sqrt(sxp * sxp + syp * syp + 1)
        if self.solid is not None:
            gzp = torch.where(self.solid, self.gz0, gzp)
        inflow = None
        if p["inflow"]:
            vin = max(-0.035, self.t / 100 * -0.035)
            hin = (abs(vin) * 0.045 / math.sqrt(0.7)) ** 0.6
            inflow = (hin, vin, min(500.0, self.t / 100 * 500) * hin / hin if hin > 0 else math.nan)
        fx0, fx1, fx2, cx, sa = self._faces(0, h0, u, v, gzp, sed, None)
        fy0, fy1, fy2, cy, sb = self._faces(1, h0, u, v, gzp, sed, inflow)
        dt = min(p["cstable"] * p["dx"] / max(sa, sb), p["maxstep"]) if max(sa, sb) > 0 else p["maxstep"]
        dt = min(dt, p["tend"] - self.t)
        dtdx = dt / p["dx"]
        if p["storm_peak"] > 0:
            x = (torch.arange(1, p["nx"] + 1, device=self.dev, dtype=torch.float64)[:, None] - 0.5) * p["dx"]
            y = (torch.arange(1, p["ny"] + 1, device=self.dev, dtype=torch.float64)[None, :] - 0.5) * p["dx"]
            r2 = (x - (p["storm_x0"] + p["storm_vx"] * self.t)) ** 2 + (y - (p["storm_y0"] + p["storm_vy"] * self.t)) ** 2
            rain = p["storm_peak"] * torch.exp(-0.5 * r2 / p["storm_radius"] ** 2)
        else:
            rain = zero + float(self.rain[int(min(math.ceil(self.t / p["rint"] + 0.01), p["rnum"])) - 1])
        # bed slope, density and debris forcing (SWEHR.c:1239-1320)
        sx, sy = self._slope(zc, 0), self._slope(zc, 1)
        root = torch.sqrt(sx * sx + sy * sy + 1)
        gz = g / root
        srcx = -g * sx / torch.sqrt(sx * sx + syp * syp + 1) * h0
        srcy = -g * sy / root * h0
        totsed0, totm0, dep0 = self.totsed, self.totm, self.dep
        rho = torch.clamp(rhow * (1 - totsed0) + rhos * totsed0, max=0.8 * rhos)
        gam = (rhos - rho) * gz * h0 * h0 / (2 * rho) * 0.5 / p["dx"]
        gx, gy = zero.clone(), zero.clone()
        gx[1:-1] = -gam[1:-1] * (totsed0[2:] - totsed0[:-2])
        gy[:, 1:-1] = -gam[:, 1:-1] * (totsed0[:, 2:] - totsed0[:, :-2])
        fail = self._failure(sx, sy, sxp, syp, gz, dep0, rho, h0)
        dfm = torch.clamp((totsed0 - 0.2) / 0.2, max=1.0)
        dfm = torch.where((h0 < 9 * p["h0"]) | (totsed0 < 0.2), zero, dfm)
        beta = -(1 - p["lambda_"]) * gz * h0 * p["frictionangle"]
        bx, by = torch.where(hu0 < 0, -beta, beta), torch.where(hv0 < 0, -beta, beta)
        # detachment and deposition (SWEHR.c:1330-1401)
        hvert = h0 * torch.sqrt(1 + sx * sx + sy * sy)
        deep = hvert > p["h0"]
        dfac = torch.where(deep, (p["h0"] / hvert) ** p["b"], one)
        Hs = torch.fmin(one, totm0 / (p["mtstar0"] * dfac))
        splash = (h0 > 10 * film) & (totsed0 < 0.6)
        man = self._manning(h0)
        q = torch.sqrt(hu0 * hu0 + hv0 * hv0)
        omega = rho * gz * (man * man * q * q / h0 ** 3.333) * q
        e3b = torch.where(splash & (omega > p["uc"]), p["af"] * (omega - p["uc"]), zero)
        e4b = torch.where(splash & (omega > p["uc2"]), p["afr"] * (omega - p["uc2"]), zero)
        e4den = (rhos - rho) / rhos * gz * h0
        vfc = (1 - torch.clamp(totsed0, max=0.99)) ** 4
        debris = (h0 > 9 * p["h0"]) & (totsed0 > p["cthreshold"])
        act = splash & ~debris
        # conservative update and Green-Ampt (SWEHR.c:1424-1452)
        h = h0 - dtdx * (fx0[1:] - fx0[:-1]) - dtdx * (fy0[:, 1:] - fy0[:, :-1]) + dt * rain
        hu = hu0 - dtdx * (fx1[1:] - fx1[:-1]) - dtdx * (fy2[:, 1:] - fy2[:, :-1]) + dt * srcx + dt * gx + dt * dfm * bx
        hv = hv0 - dtdx * (fx2[1:] - fx2[:-1]) - dtdx * (fy1[:, 1:] - fy1[:, :-1]) + dt * srcy + dt * gy + dt * dfm * by
        zf = self.vinf / (p["thetas"] - p["theta0"])
        infl = torch.minimum(h - film, dt * self.ks * (zf + p["hf"] + h) / zf)
        vinf = self.vinf + infl
        h = h - infl
        # classes (SWEHR.c:1454-1511)
        z, totm, dep, ch = zc, zero, zero, zero
        Un, Mn = [], []
        for k in range(S):
            d, pf, M0 = self.ds[k], self.pf[k], self.M[k]
            fx, fy = fx0 * cx[k], fy0 * cy[k]
            uf = self.U[k] - dtdx * (fx[1:] - fx[:-1]) - dtdx * (fy[:, 1:] - fy[:, :-1])
            E1 = torch.where(act, (1 - Hs) * pf * p["a"] * rain * dfac, zero)
            shallow = h < 10 * film
            E2 = torch.where(act & (totm0 > 1e-8) & (M0 > 1e-8), Hs * M0 / totm0 * p["ad"] * rain, zero) * dfac
            E3 = torch.where(act & (h0 > d), (1 - Hs) * pf * p["F"] / p["J"] * e3b, zero)
            E4 = torch.where(act & (h0 > d) & (totm0 > 1e-6) & (M0 > 0),
                             (1 - p["betabedload"]) * Hs * M0 / totm0 * p["F"] / e4den * e4b, zero)
            A = 13.95 * p["nu"] / d
            c = 1.09 * (rhos / rhow - 1) * gz * d
            VF = c / (torch.sqrt(A * A + c) + A) * vfc
            for limit in (1e-4, 2e-3):
                if d > limit:
                    part = 2e-3 + torch.clamp(h0 - 3 * p["h0"], min=0) * (VF - 2e-3) / (6 * p["h0"])
                    VF = torch.where(h0 < 9 * p["h0"], part, VF)
            VF = torch.where(debris, zero, VF)
            dec = torch.exp(-VF / h * (0.5 * dt))
            un = dec * (dec * uf + dt * (E1 + E3) + torch.fmin(M0, dt * (E2 + E4)))
            ch = torch.where(shallow, ch, uf)
            Mk = torch.where(shallow, M0 + dt * E1 + uf, M0 + dt * (E1 + E3) - (un - uf))
            un = torch.where(shallow, zero, un)
            z = torch.where(shallow, z, z - (un - uf) / porod)
            if fail is not None:
                f = fail & ~shallow
                z = torch.where(f, z - 0.99 * Mk / porod, z)
                un = torch.where(f, un + 0.99 * Mk, un)
                totm, dep = torch.where(f, zero, totm), torch.where(f, zero, dep)
                Mk = torch.where(f, 0.01 * Mk, Mk)
            h = h + (un - ch) / porod
            totm, dep = totm + Mk, dep + Mk / rhos
            Un.append(un)
            Mn.append(Mk)
        # concentrations, the dry clamp and friction (SWEHR.c:1513-1588)
        wet = h > film
        totsed = zero
        for k in range(S):
            totsed = totsed + Un[k] / h / rhos
            z = torch.where(wet, z, z + Un[k] / porod)
            Mn[k] = torch.where(wet, Mn[k], Mn[k] + Un[k])
            Un[k] = torch.where(wet, Un[k], zero)
        totsed = torch.where(wet, totsed, zero)
        h = torch.where(wet, h, zero + film)
        hu, hv = torch.where(wet, hu, zero), torch.where(wet, hv, zero)
        man = self._manning(h)
        fr = 1 + dt * (man * man * gz * torch.sqrt(hu * hu + hv * hv) / h ** 2.333)
        hu, hv = hu / fr, hv / fr
        if self.solid is not None:             # SWEHR.c:1233, 1421, 1566-1574
            s = self.solid
            h, hu, hv = (torch.where(s, zero, a) for a in (h, hu, hv))
            Un = [torch.where(s, zero, a) for a in Un]
            Mn = [torch.where(s, b, a) for a, b in zip(Mn, self.M)]
            vinf, z = torch.where(s, self.vinf, vinf), torch.where(s, zc, z)
            totm, dep, totsed = (torch.where(s, b, a) for a, b in ((totm, totm0), (dep, dep0), (totsed, totsed0)))
        self.h, self.hu, self.hv, self.vinf, self.U, self.M = h, hu, hv, vinf, Un, Mn
        self.totm, self.dep, self.totsed, self.zp, self.z = totm, dep, totsed, zc, z
        self.t += dt

    def _manning(self, h):
        p = self.p
        return torch.where(h <= p["hcfriction"], p["roughness"] * (h / p["hcfriction"]) ** p["depthdependentexponent"],
                           torch.full_like(h, p["roughness"]))

    def _failure(self, sx, sy, sxp, syp, gz, dep, rho, h):
        """Slope failure of the deposit (SWEHR.c:1292-1312)."""
        p = self.p
        rho0 = p["rhow"] * p["phi"] + p["rhos"] * (1 - p["phi"])
        own_x, own_y, sxc, syc = sx, sy, sx, sy
        if self.solid is not None:
            s = self.solid
            sxp, syp = torch.where(s, self.sx0, sxp), torch.where(s, self.sy0, syp)
            sxc, syc = torch.where(s, self.sx0, sxc), torch.where(s, self.sy0, syc)

        def cos(a):
            return 1 / torch.sqrt(1 + a * a)

        def term(dim, own, before, now):
            tr = (lambda a: a) if dim == 0 else (lambda a: a.t())
            d, o, b, n = tr(dep), cos(tr(own)), cos(tr(before)), cos(tr(now))
            up = torch.cat([d[1:] * b[1:], d[-1:] * o[-1:]])
            dn = torch.cat([d[:1] * o[:1], d[:-1] * n[:-1]])
            f = tr(dep * rho0 * gz) * 0.5 / p["dx"] * (up - dn)
            s = tr(own)
            f = torch.where(f * s > 0, -f.abs(), f)
            f = torch.where(f * s < 0, f.abs(), f)
            return f if dim == 0 else f.t()

        w = rho0 * gz * dep + rho * gz * h
        lhs = w * sy.abs() / torch.sqrt(1 + sy * sy)
        rhs = p["cohesion"] + (w * cos(sy) - p["rhow"] * gz * (dep + h)) * p["frictionangle"]
        fail = (lhs > rhs + term(0, own_x, sxp, sxc)) | (lhs > rhs + term(1, own_y, syp, syc))
        return fail if bool(fail.any()) else None

    def speed(self):
        wet = self.h > self.p["hfilm"]
        v = torch.sqrt(self.hu * self.hu + self.hv * self.hv) / self.h
        return torch.where(wet, v, torch.zeros_like(v))


def _exact_fields(case, seed, names, tend=None):
    made, snap = _inputs(case, seed)
    if tend is not None:
        made.params["tend"] = tend
    e = _Exact(made, snap)
    for _ in range(case["steps"]):
        e.step()
    have = {"z": e.z, "h": e.h, "vel": e.speed(), "totsed": e.totsed, "totm": e.totm}
    return {n: have[n].contiguous().cpu().numpy() for n in names}


def exact(case, seed):
    if case["kind"] == "domain":
        out = _exact_fields(case, seed, FRAME)
        if case["budget"]:
            out["budget"] = None
        return out
    return [_exact_fields(sub, sub_seed, RESULT, tend=36000.0) for sub, sub_seed in _scenarios(case, seed)]
