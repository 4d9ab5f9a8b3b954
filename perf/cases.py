"""The work that a user of this framework has it do, as cases to be timed.

Five kinds of call, each through the public entry points:

  static  impz_deposit_static on the caller's device buffers (a host code with
          its own memory pool, or a timed loop of another program)
  step    the reference's per-step surface (map_half, sc_prepare, deposit,
          poisson, kick, map_half, moments), as the Fortran driver calls it
  run     one job: upload of the host's particles, a whole lattice, the moment
          records back, and where a user dumps phase space the particles too
  scan    run_batch over independent bunches of uneven size
  serve   jobs submitted to the serving loop and waited for

A pass starts from the particles the host holds (pinned, as the benchmark's
end-to-end job has them), so every pass does the same work.  Moments come back
as means over the bunch, in units of its rms sizes at the start.

exact() restates the step in plain torch at 64 bits: maps, z->t transform,
cloud-in-cell deposit, Hockney's convolution with the integrated Green
function, finite-difference field, kick, read-in wake and the Lorentz
integrator's update.
"""
import ctypes
import importlib.util
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
CLIGHT = 299792458.0
PROTON, ELECTRON, AMU = 938.27208816e6, 0.51099895000e6, 931.49410242e6


def package():
    if "impz_b200" not in sys.modules:
        pkg = os.path.join(ROOT, "impact-z_b200")
        spec = importlib.util.spec_from_file_location(
            "impz_b200", os.path.join(pkg, "__init__.py"), submodule_search_locations=[pkg])
        mod = importlib.util.module_from_spec(spec)
        sys.modules["impz_b200"] = mod
        spec.loader.exec_module(mod)
    return sys.modules["impz_b200"]


# ---------------------------------------------------------------------------
# the cases
def _case(kind, beam, form, n, grid, steps, **more):
    nx, ny, nz = grid
    c = dict(kind=kind, beam=beam, form=form, n=n, nx=nx, ny=ny, nz=nz, steps=steps, lattice="fodo",
             gradient=20.0, integrator=1, wake=0, dump=False, grids=False, bunches=1, nmin=n)
    c.update(more)
    return c


def listed():
    return [
        # the smallest call: a few thousand particles per rank deposited between a host code's
        # own kernels; launches and latency are all there is
        _case("static", "proton", "fp64", 20_000, (32, 32, 64), 1, name="static_small"),
        # the same for a full bunch in the order the host code happens to hold it
        _case("static", "proton", "fp64", 4_000_000, (64, 64, 128), 1, name="static_large"),
        # the Fortran driver on the 32x32x64 benchmark beam, looking at every grid it computes
        _case("step", "proton", "fp64", 100_003, (32, 32, 64), 1, grids=True, name="step_fp64_grids"),
        # the Fortran driver with the data left on the GPU, four steps of a large beam
        _case("step", "proton", "fp32", 1_000_001, (64, 64, 128), 4, name="step_fp32_resident"),
        # the small benchmark job as written (160 steps, plain FP64), phase space dumped at the end
        _case("run", "proton", "fp64", 100_000, (32, 32, 64), 160, dump=True, name="run_fodo_1e5_fp64"),
        # the headline beam in the FP32-convolution form
        _case("run", "proton", "fp32", 4_000_000, (64, 64, 128), 100, name="run_fodo_4e6_fp32"),
        # the plain FP64 form on the headline grid, an odd particle count
        _case("run", "proton", "fp64", 1_000_001, (64, 64, 128), 60, gradient=15.0,
              name="run_fodo_1e6_fp64"),
        # the modulated electron bunch: long grid, drift and chicane, the full map set
        _case("run", "electron", "fp32", 20_000_000, (64, 64, 2048), 36, lattice="chicane",
              name="run_chicane_2e7"),
        # Lorentz integrator with a read-in wake
        _case("run", "linac", "fp32", 500_000, (32, 32, 128), 40, lattice="linac", integrator=2,
              wake=1, gradient=10.0, name="run_lorentz_wake"),
        # two charge states of an ion beam through K-map quadrupoles
        _case("run", "ion", "fp32", 300_001, (32, 32, 64), 48, lattice="kquad", gradient=8.0,
              name="run_charge_states"),
        # a parameter scan: independent bunches of 1e4 to 2e6 particles on the three grids
        _case("scan", "proton", "fp32", 2_000_000, (64, 64, 128), 40, bunches=24, nmin=10_000,
              name="scan_24"),
        # served jobs of uneven size and length
        _case("serve", "proton", "fp32", 1_000_000, (64, 64, 128), 64, bunches=8, nmin=10_000,
              name="serve_8"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["static", "step", "run", "run", "run", "run", "scan", "serve"])
    grid = (rng.choice([8, 16, 32, 64]), rng.choice([8, 16, 32, 64]), rng.choice([16, 32, 64, 128, 256]))
    grad = round(rng.uniform(10.0, 20.0), 3)
    form = rng.choice(["fp64", "fp32"])
    if kind == "static":
        return _case("static", "proton", "fp64", _log(rng, 1e3, 4e6), grid, 1)
    if kind == "step":
        return _case("step", "proton", form, _log(rng, 1e4, 2e6), grid, rng.randint(1, 4),
                     gradient=grad, grids=form == "fp64" and rng.random() < 0.5)
    if kind == "scan":
        hi = _log(rng, 1e5, 1e6)
        return _case("scan", "proton", form, hi, grid, rng.randint(10, 40), gradient=grad,
                     bunches=rng.randint(3, 24), nmin=max(5000, hi // 100))
    if kind == "serve":
        hi = _log(rng, 1e5, 1e6)
        return _case("serve", "proton", form, hi, grid, rng.randint(20, 64), gradient=grad,
                     bunches=rng.randint(2, 8), nmin=max(5000, hi // 100))
    what = rng.choice(["fodo", "fodo", "fodo", "chicane", "linac", "kquad"])
    if what == "chicane":
        grid = (rng.choice([32, 64]), rng.choice([32, 64]), rng.choice([256, 512, 1024, 2048]))
        return _case("run", "electron", form, _log(rng, 2e5, 1e7), grid, rng.randint(30, 40),
                     lattice="chicane")
    if what == "linac":
        return _case("run", "linac", form, _log(rng, 2e4, 1e6), grid, rng.randint(16, 48),
                     lattice="linac", integrator=rng.choice([1, 2]), wake=rng.randint(0, 1),
                     gradient=round(rng.uniform(4.0, 10.0), 3))
    if what == "kquad":
        return _case("run", "ion", form, _log(rng, 2e4, 1e6), grid, rng.randint(16, 48),
                     lattice="kquad", gradient=round(rng.uniform(4.0, 10.0), 3))
    n = _log(rng, 1e4, 4e6)
    return _case("run", "proton", form, n, grid, rng.randint(16, 100), gradient=grad,
                 dump=n < 200_000 and rng.random() < 0.5)


# ---------------------------------------------------------------------------
# inputs
def _normal(gen, n, k=6, cut=4.0):
    z = torch.randn((k, n), generator=gen, device="cuda", dtype=torch.float64)
    bad = z.abs() > cut
    while bool(bad.any()):
        z[bad] = torch.randn(int(bad.sum()), generator=gen, device="cuda", dtype=torch.float64)
        bad = z.abs() > cut
    return z


BEAMS = {  # mass, charge, kinetic energy [eV], current [A], Scfreq [Hz]
    "proton": (PROTON, 1.0, 2.5e6, 0.030, 402.5e6),
    "electron": (ELECTRON, -1.0, 250e6 - ELECTRON, 100.0, 1.3e9),
    "linac": (ELECTRON, -1.0, 98.169272e6, 1.3, 1.3e9),
    "ion": (238 * AMU, 29.0, 0.5e6 * 238, 2.5e-4, 80.5e6),
}
SIGMAS = {  # rms x, y [m], x', y' [rad], phase [rad], energy [eV]
    "proton": (1e-3, 1e-3, math.radians(5.0), 50e3),
    "linac": (0.5e-3, 0.05e-3, math.radians(1.0), 50e3),
    "ion": (2e-3, 0.5e-3, math.radians(5.0), 2e4),
}


def _beam(name, n, seed, current=None):
    """Pts1 (n, 9) on the GPU and the beam's constants."""
    gen = torch.Generator(device="cuda").manual_seed(seed)
    mass, charge, ekin, cur, freq = BEAMS[name]
    cur = cur if current is None else current
    gam = 1.0 + ekin / mass
    gb = math.sqrt(gam * gam - 1.0)
    xl = CLIGHT / (2 * math.pi * freq)
    pts = torch.empty((n, 9), device="cuda", dtype=torch.float64)
    if name == "electron":
        # 1 mm flat top, 1 % density modulation at 10 um (rejection sampled)
        got = torch.empty(0, device="cuda", dtype=torch.float64)
        while got.numel() < n:
            u = torch.rand((2, n + n // 20 + 1024), generator=gen, device="cuda", dtype=torch.float64)
            s = (u[0] - 0.5) * 1e-3
            keep = u[1] * 1.01 < 1 + 0.01 * torch.cos(2 * math.pi * s / 10e-6)
            got = torch.cat([got, s[keep]])
        t = _normal(gen, n, 5)
        sx, sp = 0.2e-3 / xl, 0.02e-3 * gb
        for c, f in enumerate((sx, sp, sx, sp)):
            pts[:, c] = t[c] * f
        pts[:, 4] = -got[:n] / (gb / gam * xl)
        pts[:, 5] = t[4] * (5e3 / mass)
    else:
        sx, sp, sph, se = SIGMAS[name]
        z = _normal(gen, n)
        for c, f in enumerate((sx / xl, sp * gb, sx / xl, sp * gb, sph, se / mass)):
            pts[:, c] = z[c] * f
    pts[:, 6] = charge / mass
    pts[:, 7] = cur / freq / n * math.copysign(1.0, charge)
    if name == "ion":  # every other particle, in effect, has one charge more
        second = torch.rand(n, generator=gen, device="cuda") < 0.4
        pts[:, 6] = torch.where(second, (charge + 1) / mass, charge / mass)
        pts[:, 7] = torch.where(second, 1.3 * cur / freq / n, cur / freq / n)
    pts[:, 8] = torch.arange(1, n + 1, device="cuda", dtype=torch.float64)
    ref = np.zeros(6)
    ref[5] = -gam
    return dict(pts=pts, current=cur, mass=mass, charge=charge, freq=freq, ref=ref)


def _lattice(case, steps, gradient):
    """[(type, length, nseg, mapstp, values)] of exactly `steps` steps."""
    if case["lattice"] == "chicane":
        # 20 m in 756 steps is the benchmark's drift; here its step length, then the four bends
        a, nb = math.radians(3.0), max(1, min(8, (steps - 6) // 5))
        bend = lambda s: (4, 0.2, nb, 1, (s * a, 0.0, 150.0, 0.01) + 5 * (0.0,))  # noqa: E731
        first = max(1, steps - 4 * nb - 3)
        d = (0, 3.5, 1, 1, (1.0,))
        return [(0, 20.0 / 756 * first, first, 1, (1.0,)), bend(1), d, bend(-1),
                (0, 0.5, 1, 1, (1.0,)), bend(-1), d, bend(1)]
    if case["lattice"] == "linac":
        pat, seg = [(0, 0.5, None), (1, 0.1, 1), (0, 0.5, None), (1, 0.1, -1)], 8
    elif case["lattice"] == "kquad":
        pat, seg = [(0, 0.1, None), (1, 0.1, 1), (0, 0.1, None), (1, 0.1, -1)], 4
    else:
        pat, seg = [(0, 0.1, None), (1, 0.1, 1), (0, 0.1, None), (1, 0.1, -1)], 4
    out, left, i = [], steps, 0
    mode = -1.0 if case["lattice"] == "kquad" else 0.0
    while left > 0:
        t, length, sign = pat[i % 4]
        k = min(seg, left)
        vals = (1.0,) if sign is None else (sign * gradient, mode, 1.0)
        out.append((t, length * k / seg, k, 1, vals))
        left -= k
        i += 1
    return out


def _members(case, seed):
    """The bunches of a case: particles, grid, gradient, current, steps each."""
    if case["kind"] not in ("scan", "serve"):
        return [dict(n=case["n"], grid=(case["nx"], case["ny"], case["nz"]), gradient=case["gradient"],
                     current=None, steps=case["steps"], seed=seed)]
    g = (case["nx"], case["ny"], case["nz"])
    grids = [g, (max(8, g[0] // 2), max(8, g[1] // 2), max(16, g[2] // 2)),
             (max(8, g[0] // 4), max(8, g[1] // 4), max(16, g[2] // 8))]
    nb, out = case["bunches"], []
    for i in range(nb):  # log-uniform counts from nmin to n, grids in turn
        u = (i + 0.5) / nb
        n = int(round(math.exp(math.log(case["nmin"]) + u * math.log(case["n"] / case["nmin"]))))
        steps = case["steps"] if case["kind"] == "scan" else max(8, case["steps"] - 5 * (i % 4))
        out.append(dict(n=n | 1, grid=grids[i % 3], gradient=case["gradient"] * (0.75 + 0.25 * u),
                        current=0.005 + 0.045 * u, steps=steps, seed=seed * 64 + i))
    return out


def _wake_table():
    z = np.linspace(0.0, 5e-3, 201)
    return np.column_stack([z, 3e13 * np.exp(-z / 1e-3), 2e15 * z, 2e15 * z])


def _pinned(pts):
    host = torch.empty(pts.shape, dtype=torch.float64, pin_memory=True)
    host.copy_(pts)
    return host.numpy()


def prepare(case, seed):
    impz = package()
    mem = _members(case, seed)
    if case["kind"] == "static":
        b = _beam(case["beam"], case["n"], seed)
        cols = [b["pts"][:, c].contiguous() for c in range(6)]
        rng = _static_box(b, mem[0]["grid"])
        nx, ny, nz = mem[0]["grid"]
        out = torch.empty((nz, ny, nx), device="cuda", dtype=torch.float64)
        args = tuple(c.data_ptr() for c in cols) + (
            case["n"], -b["ref"][5], 1.0, 1.0, b["freq"], float(b["pts"][0, 7]),
            rng.ctypes.data_as(ctypes.POINTER(ctypes.c_double)), nx, ny, nz, out.data_ptr(), None)
        torch.cuda.synchronize()
        return dict(kind="static", lib=impz.lib(), args=args, out=out, keep=(cols, rng))
    form = impz.FORM_FP64 if case["form"] == "fp64" else impz.FORM_FP32CONV
    s = dict(kind=case["kind"], impz=impz, case=dict(case), members=[])
    for m in mem:
        b = _beam(case["beam"], m["n"], m["seed"], m["current"])
        pts = _pinned(b["pts"])
        lat = [impz.elem(t, length, nseg, mapstp, vals)
               for t, length, nseg, mapstp, vals in _lattice(case, m["steps"], m["gradient"])]
        h = dict(pts=pts, ref=b["ref"], beam={k: b[k] for k in ("current", "mass", "charge", "freq")},
                 lattice=lat, grid=m["grid"], form=form)
        if case["kind"] != "serve":
            h["bunch"] = impz.Bunch(pts, b["current"], b["mass"], b["charge"], b["freq"], b["ref"],
                                    m["grid"], form=form, track_ids=case["dump"],
                                    species=case["beam"] == "ion")
            if case["integrator"] == 2:
                h["bunch"].set_integrator(2)
            if case["wake"]:
                h["bunch"].wake(_wake_table(), 1.0, True)
        s["members"].append(h)
    if case["kind"] == "serve":
        s["server"] = impz.Server(budget_bytes=160e9, max_active=64)
    torch.cuda.synchronize()
    return s


# ---------------------------------------------------------------------------
# one pass
LOW = {"x": (0, 1, 6, 7, 12), "y": (2, 3, 8, 9, 13), "z": (4, 5, 10, 11, 14)}
HIGH = {"x": (15, 16, 17, 18, 27, 28, 29, 30, 31), "y": (19, 20, 21, 22, 32, 33, 34, 35, 36),
        "z": (23, 24, 25, 26)}
POWERS = [(1, 0), (0, 1), (2, 0), (0, 2), (1, 1), (3, 0), (4, 0), (0, 3), (0, 4), (1, 2), (1, 3), (2, 1),
          (2, 2), (3, 1)]  # of (position, momentum), in the order of LOW + HIGH


def _moments(recs):
    """All the moments of the records, as means over the bunch in units of its rms sizes at
    the start: per plane the first and second ones, and the third and fourth; the maxima;
    counts and current.  Records of several bunches one after another."""
    low, high, top, rest = {k: [] for k in LOW}, {k: [] for k in LOW}, [], []
    for r in recs:
        m = r[:, :37] / r[:, 44:45]
        sig = np.sqrt((r[0, 6:12] / r[0, 44]))
        for d, k in enumerate(LOW):
            cols = LOW[k] + HIGH[k]
            unit = [sig[2 * d] ** a * sig[2 * d + 1] ** b for a, b in POWERS[:len(cols)]]
            v = m[:, cols] / np.array(unit)
            low[k].append(v[:, :5])
            high[k].append(v[:, 5:])
        top.append(np.concatenate([r[:, 37:43] / sig, r[:, 43:44] / sig[0] ** 2], axis=1))
        rest.append(r[:, 44:47])
    out = {"second_" + k: np.concatenate(v) for k, v in low.items()}
    out.update({"fourth_" + k: np.concatenate(v) for k, v in high.items()})
    rest = np.concatenate(rest)
    out.update({"maxima": np.concatenate(top), "npt": rest[:, 0], "nlocal": rest[:, 1],
                "current": rest[:, 2]})
    return out


def run(s):
    if s["kind"] == "static":
        rc = s["lib"].impz_deposit_static(*s["args"])
        if rc:
            raise RuntimeError("impz_deposit_static: %d" % rc)
        return s["out"]
    return {"step": _run_step, "run": _run_job, "scan": _run_scan, "serve": _run_serve}[s["kind"]](s)


def _run_step(s):
    h, case = s["members"][0], s["case"]
    b, out, recs, z = h["bunch"], {}, [], 0.0
    b.upload(h["pts"], h["beam"]["current"], h["ref"])
    e = h["lattice"][0]
    tau = e.length / e.nseg / 2
    ih = 0
    for j in range(case["steps"]):
        z, ih = b.map_half(e, 0.0, z, tau, j + 1, ih)
        nptot, ptrange, box, msize = b.sc_prepare(1.0, 1.0)
        rho, counts = b.deposit(want_rho=case["grids"], want_counts=case["grids"])
        phi = b.poisson(want_phi=case["grids"])
        eg = b.kick(2 * tau, want_e=case["grids"])
        z, ih = b.map_half(e, 0.0, z, tau, j + 1, ih)
        recs.append(b.moments())
    out = _moments([np.array(recs)])
    out.update({"ptrange": ptrange, "range": box, "msize": msize})
    if case["grids"]:
        out.update({"rho": rho, "counts": counts, "phi": phi, "e": eg})
    return out


def _run_job(s):
    h = s["members"][0]
    b = h["bunch"]
    b.upload(h["pts"], h["beam"]["current"], h["ref"])
    recs, zs = b.run(h["lattice"])
    out = _moments([recs])
    out["z"] = zs
    if s["case"]["dump"]:  # phase space in the order of the input
        p = b.download()
        q = np.empty_like(p)
        q[p[:, 8].astype(np.int64) - 1] = p
        out.update({"phase_space%d" % c: q[:, c] for c in range(6)})
    return out


def _run_scan(s):
    impz, mem = s["impz"], s["members"]
    for h in mem:
        h["bunch"].upload(h["pts"], h["beam"]["current"], h["ref"])
    got = impz.run_batch([h["bunch"] for h in mem], [h["lattice"] for h in mem])
    return _moments([r for r, _ in got])


def _run_serve(s):
    jobs = [s["server"].submit(h["pts"], grid=h["grid"], refptcl=h["ref"], lattice=h["lattice"],
                               form=h["form"], **h["beam"]) for h in s["members"]]
    return _moments([s["server"].wait(j)[0] for j in jobs])


# ---------------------------------------------------------------------------
# what a pass cannot do without
def work(case):
    bytes_, flops = 0.0, 0.0
    for m in _members(case, 0):
        g = float(m["grid"][0] * m["grid"][1] * m["grid"][2])
        if case["kind"] == "static":
            bytes_ += 48.0 * m["n"] + 8.0 * g
            flops += 120.0 * m["n"]
            continue
        f64 = case["form"] == "fp64"
        # a step: positions for the deposit, the state read and written; charge, doubled-grid
        # convolution, field
        step = 120.0 * m["n"] + (16.0 + (152.0 if f64 else 76.0) + (8.0 if f64 else 4.0)) * g
        bytes_ += 144.0 * m["n"] + step * m["steps"]
        flops += m["steps"] * (450.0 * m["n"] + g * (100.0 + 8 * 5.0 * 2 * math.log2(8 * g)))
        if case["grids"]:
            bytes_ += 44.0 * g
        if case["dump"]:
            bytes_ += 72.0 * m["n"]
    return {"bytes": bytes_, "flops": flops}


def tolerance(case):
    """About four times what was seen between the framework and the 64-bit restatement, or
    between runs with the sums in another order."""
    if case["kind"] == "static":
        return {"rel": 2e-12, "max": 2e-10}
    if case["form"] == "fp64":
        return {"rel": 4e-12, "max": 1e-10} if case["kind"] == "step" else {"rel": 1e-10, "max": 1e-8}
    if case["lattice"] == "chicane":  # one outermost particle's energy decides the maxima
        return {"rel": 1.5e-5, "max": 1e-4}
    return {"rel": 2e-6, "max": 2e-5}


# ---------------------------------------------------------------------------
# the same in plain torch, 64 bits
PILC = float(np.float32(2.0) * np.float32(math.asin(1.0)))  # the reference's single-precision pi
E7 = float(np.float32(1.0e-7))


def _tframe(p, gam, xl):
    x, px, y, py, ph, pt = p
    if float(ph.abs().max()) >= PILC:
        k = torch.trunc(ph / PILC)
        ph = ph - k * PILC - torch.fmod(k, 2) * PILC
    rcp = 1.0 / (gam - pt)
    bet2 = 1.0 - rcp * rcp * (1.0 + px * px + py * py)
    zt = -(gam * bet2.abs().sqrt() * ph * xl)
    return (x - px * ph * rcp) * xl, (y - py * ph * rcp) * xl, zt, rcp, bet2


def _box(lo, hi, grid):
    out, h = [], []
    for d in range(3):
        eps = float(np.float32(1.0) / (np.float32(grid[d]) - np.float32(3.0)))
        a, b = lo[d] - eps * (hi[d] - lo[d]), hi[d] + eps * (hi[d] - lo[d])
        out += [a, b]
        h.append((b - a) / (grid[d] - 1))
    return out, h


def _static_box(b, grid):
    p = [b["pts"][:, c] for c in range(6)]
    xl = CLIGHT / (2 * math.pi * b["freq"])
    xt, yt, zt, _, _ = _tframe(p, -b["ref"][5], xl)
    lo, hi = [float(v.min()) for v in (xt, yt, zt)], [float(v.max()) for v in (xt, yt, zt)]
    return np.array(_box(lo, hi, grid)[0])


def _cic(pos, box, h):
    i, w = [], []
    for d in range(3):
        k = ((pos[d] - box[2 * d]) / h[d] + 1.0).to(torch.int64)
        i.append(k - 1)
        w.append(((box[2 * d] - pos[d]) + k.double() * h[d]) / h[d])
    return i, w


CORNERS = [(a, b, c) for a in (0, 1) for b in (0, 1) for c in (0, 1)]


def _corner(i, w, grid, a, b, c):
    node = (i[0] + a) + grid[0] * ((i[1] + b) + grid[1] * (i[2] + c))
    wt = (1 - w[0] if a else w[0]) * (1 - w[1] if b else w[1]) * (1 - w[2] if c else w[2])
    return node, wt


def _deposit(i, w, grid, weight):
    rho = torch.zeros(grid[0] * grid[1] * grid[2], device="cuda", dtype=torch.float64)
    for a, b, c in CORNERS:
        node, wt = _corner(i, w, grid, a, b, c)
        rho.index_add_(0, node, wt * weight)
    return rho


def _green(grid, h):
    v = [(torch.arange(grid[d] + 2, device="cuda", dtype=torch.float64) - 0.5) * h[d] for d in range(3)]
    x, y, z = v[0][None, None, :], v[1][None, :, None], v[2][:, None, None]
    r = (x * x + y * y + z * z).sqrt()
    f = y * z * torch.log(x + r) + x * z * torch.log(y + r) + x * y * torch.log(z + r)
    f = f - 0.5 * (z * z * torch.atan(x * y / (z * r)) + y * y * torch.atan(x * z / (y * r)) +
                   x * x * torch.atan(y * z / (x * r)))
    f = f / (h[0] * h[1] * h[2])
    for d in (2, 1, 0):
        f = f.diff(dim=d)
    for d in range(3):  # even about 0 and about the doubled grid's middle
        n = f.shape[d] - 1
        f = torch.cat([f, f.narrow(d, 1, n - 1).flip(d)], dim=d)
    return f


def _potential(rho, grid, h):
    nx, ny, nz = grid
    shape = (2 * nz, 2 * ny, 2 * nx)
    g = torch.fft.rfftn(_green(grid, h))
    r = torch.fft.rfftn(rho.view(nz, ny, nx), s=shape)
    return torch.fft.irfftn(g * r, s=shape)[:nz, :ny, :nx].contiguous()


def _field(phi, h):
    out = []
    for d, k in ((2, 0), (1, 1), (0, 2)):
        n = phi.shape[d]
        inner = (phi.narrow(d, 0, n - 2) - phi.narrow(d, 2, n - 2)) * (0.5 / h[k])
        first = (phi.narrow(d, 0, 1) - phi.narrow(d, 1, 1)) / h[k]
        last = (phi.narrow(d, n - 2, 1) - phi.narrow(d, n - 1, 1)) / h[k]
        out.append(torch.cat([first, inner, last], dim=d).reshape(-1))
    return out


def _kick_consts(c, gam, cur):
    bet = math.sqrt(gam * gam - 1.0) / gam
    gb = gam * bet
    brho = gb / (CLIGHT * c["charge"]) * c["mass"]
    perv = 2.0 * cur * CLIGHT * CLIGHT * E7 / (brho * (bet * CLIGHT) ** 2 * gam * gam)
    xl = CLIGHT / (2 * math.pi * c["freq"])
    xy = 0.5 * perv * gb * (bet * xl) * 2 * math.pi / (cur / c["freq"])
    return xy, bet * xy * gam * gam


def _wake_planes(c, gam, cur, npt, xt, yt, zt, box, nz, table):
    """The read-in wake's (x, y, z) field per plane (raw)."""
    hz0 = (box[5] - box[4]) / (nz - 1)
    k = ((zt - box[4]) / hz0 + 1).to(torch.int64)
    ab = ((box[4] - zt) + k.double() * hz0) / hz0
    line = torch.zeros((3, nz), device="cuda", dtype=torch.float64)
    for q, v in enumerate((torch.ones_like(xt), xt, yt)):
        line[q].index_add_(0, k - 1, ab * v)
        line[q].index_add_(0, k, (1 - ab) * v)
    hz = hz0 / gam
    d = line[0] * (cur / c["freq"] / npt / hz * math.copysign(1.0, c["charge"]))
    mean = torch.where(line[0] != 0, line[1:] / line[0], torch.zeros_like(line[1:]))
    t = torch.tensor(table, device="cuda")
    hw, zz = table[1, 0] - table[0, 0], torch.arange(nz, device="cuda", dtype=torch.float64) * hz
    iw = (zz / hw + 1).to(torch.int64)
    wt = iw.double() * hw - zz
    pad = torch.cat([t[:, 1:], torch.zeros((nz + 8 + int(iw.max()), 3), device="cuda", dtype=torch.float64)])
    g = (pad[iw - 1] * wt[:, None] + pad[iw] * (1 - wt)[:, None]).T  # rows z, x, y
    m = torch.arange(nz, device="cuda")
    lag = m[None, :] - m[:, None]
    far = lag > 0
    conv = lambda src, gr: (torch.where(far, gr[lag.clamp(min=0)], gr.new_zeros(())) * src[None, :]).sum(1)  # noqa: E731
    ez = -(0.5 * g[0][0] * d + conv(d, g[0])) * hz
    return conv(d * mean[0], g[1]) * hz, conv(d * mean[1], g[2]) * hz, ez


def _drift(p, gam, tau, xl):
    x, px, y, py, ph, pt = p
    d = pt - gam
    r = (d * d - 1.0 - px * px - py * py).sqrt()
    beta0 = math.sqrt(gam * gam - 1.0) / gam
    return [x + px * tau / r / xl, px, y + py * tau / r / xl, py,
            ph - (1.0 / beta0 + d / r) * tau / xl, pt]


def _quad(p, gam, tau, xl, k0):
    """Thick linear quadrupole about the reference momentum."""
    x, px, y, py, ph, pt = p
    gb = math.sqrt(gam * gam - 1.0)
    out = []
    for u, pu, k in ((x, px, k0), (y, py, -k0)):
        r = math.sqrt(abs(k))
        cs, sn = (math.cos(r * tau), math.sin(r * tau)) if k > 0 else (math.cosh(r * tau), math.sinh(r * tau))
        out += [cs * u + sn / r / (gb * xl) * pu, -math.copysign(r, k) * sn * gb * xl * u + cs * pu]
    return out + [ph + tau / (xl * gb ** 3) * pt, pt]


def _kquad(p, gam, tau, xl, k0, qm_ratio):
    x, px, y, py, ph, pt = p
    g = gam - pt
    betaz = (g * g - 1.0 - px * px - py * py).sqrt() / g
    gb = (g * g - 1.0).sqrt()
    gb0 = math.sqrt(gam * gam - 1.0)
    ks = qm_ratio * gb0 / gb * k0
    r = ks.abs().sqrt()
    a = r * tau
    foc = (torch.cos(a), torch.sin(a) / r, -torch.sin(a) * r)
    dfc = (torch.cosh(a), torch.sinh(a) / r, torch.sinh(a) * r)
    mx, my = (foc, dfc) if k0 > 0 else (dfc, foc)
    return [mx[0] * x + mx[1] * px / gb / xl, gb * xl * mx[2] * x + mx[0] * px,
            my[0] * y + my[1] * py / gb / xl, gb * xl * my[2] * y + my[0] * py,
            ph + (1.0 / betaz - gam / gb0) * tau / xl, pt]


def _pole(p, gam, xl, h0, qm0, qm):
    """Entrance or exit pole face of a sector bend without face angle: the
    second-order terms in the bend's curvature (the two faces differ in sign)."""
    x, px, y, py, ph, pt = p
    beta = math.sqrt(1.0 - 1.0 / (gam * gam))
    gb = beta * gam
    gn = gam - pt
    pz = (gn * gn - 1.0 - px * px - py * py).sqrt()
    X, xp, Y, yp = x * xl, px / pz, y * xl, py / pz
    s = 1.0 if h0[1] == "in" else -1.0
    h = h0[0]
    a0 = X + s * 0.5 * h * Y * Y
    a2 = Y
    a1 = xp
    a3 = yp - s * h * xp * Y
    pz = (gn * gn - 1.0).sqrt() / (a1 * a1 + a3 * a3 + 1).sqrt()
    return [a0 / xl, a1 * pz, a2 / xl, a3 * pz, ph, pt]


def _sector(p, gam, xl, h0, length, qm0, qm):
    x, px, y, py, ph, pt = p
    beta = math.sqrt(1.0 - 1.0 / (gam * gam))
    gb = beta * gam
    rho, th = 1.0 / h0, length * h0
    st, ct, sh = math.sin(th), math.cos(th), math.sin(th / 2)
    gi = gam - pt
    gbi = (gi * gi - 1.0).sqrt()
    pz = (gbi * gbi - px * px - py * py).sqrt()
    X, xp, Y, yp = x * xl, px / pz, y * xl, py / pz
    z0 = -(ph * beta * xl)
    eta = -(pt / beta / gb)
    a0 = (ct * X + rho * st * xp + rho * (1 - ct) * eta - st * st / (2 * rho) * X * X + st * ct * X * xp
          + st * st * X * eta + rho * ct * sh * sh * xp * xp - rho * st * (ct - 1) * xp * eta
          - 0.5 * rho * st * st * eta * eta + 0.5 * rho * (ct - 1) * yp * yp)
    a1 = (-st / rho * X + ct * xp + st * eta + st / rho * X * eta - 0.5 * st * xp * xp
          - st * eta * eta - 0.5 * st * yp * yp)
    a2 = Y + length * yp + st * X * yp + 2 * rho * sh * sh * xp * yp + rho * (th - st) * yp * eta
    a4 = (-st * X - rho * (1 - ct) * xp + z0 + rho * (st - beta * beta * th) * eta
          - 0.5 * rho * st * (xp * xp + yp * yp) + rho * (ct - 1) * xp * eta)
    pz = gbi / (a1 * a1 + yp * yp + 1).sqrt()
    return [a0 / xl, a1 * pz, a2 / xl, yp * pz, -a4 / xl / beta, pt]


def _lorentz(p, e, gam, tau, xl, c, grad, wake, qm):
    """The Lorentz integrator's implicit momentum update, twice iterated."""
    x, px, y, py, ph, pt = p
    sc, beta = CLIGHT * CLIGHT * E7, math.sqrt(gam * gam - 1.0) / gam
    ex, ey, ez = (sc * e[q] + wake[q] for q in range(3))
    bx = -beta / CLIGHT * sc * e[1] + grad * y * xl
    by = beta / CLIGHT * sc * e[0] + grad * x * xl
    f = tau * qm
    pz = ((gam - pt) ** 2 - 1.0 - px * px - py * py).sqrt()
    q1, q2, q3 = px, py, pt
    for _ in range(2):
        a13, a23 = ex * f / 2 / pz, ey * f / 2 / pz
        b1 = px - a13 * pt + gam * ex * f / pz - CLIGHT * by * f
        b2 = py - a23 * pt + gam * ey * f / pz + CLIGHT * bx * f
        b3 = -a13 * px - a23 * py + pt - ez * f
        det = 1 - a13 * a13 - a23 * a23
        q1 = ((1 - a23 * a23) * b1 + a13 * a23 * b2 - a13 * b3) / det
        q2 = (a13 * a23 * b1 + (1 - a13 * a13) * b2 - a23 * b3) / det
        q3 = (-a13 * b1 - a23 * b2 + b3) / det
        s = (gam - q3) ** 2 - 1.0 - q1 * q1 - q2 * q2
        pz = torch.where(s > 0, 0.5 * pz + 0.5 * s.clamp(min=0).sqrt(), pz)
    return [x, q1, y, q2, ph, q3]


def _drift2(p, gam, tau, xl):
    """The Lorentz integrator's drift by tau / 2."""
    x, px, y, py, ph, pt = p
    g = gam - pt
    pz = (g * g - 1.0 - px * px - py * py).sqrt()
    beta = math.sqrt(1.0 - 1.0 / gam / gam)
    return [x + 0.5 * tau * px / (xl * pz), px, y + 0.5 * tau * py / (xl * pz), py,
            ph + 0.5 * tau * (g / (xl * pz) - 1.0 / (beta * xl)), pt]


def _record(p, npt, cur):
    x, px, y, py, z, pz = p
    v = [x, px, y, py, z, pz, x * x, px * px, y * y, py * py, z * z, pz * pz, x * px, y * py, z * pz]
    for q in (x, px, y, py):
        v += [q ** 3, q ** 4]
    v += [(z ** 3).abs(), z ** 4, pz ** 3, pz ** 4]
    for a, b in ((x, px), (y, py)):
        v += [a * b * b, a * b ** 3, a * a * b, a * a * b * b, a ** 3 * b]
    r = [q.sum() for q in v] + [q.abs().max() for q in p] + [(x * x + y * y).max()]
    n = float(x.numel())
    return np.concatenate([torch.stack(r).cpu().numpy(), [npt, n, cur, 0.0]])


def _solve(p, c, grid, gam, cur, table):
    """One space-charge solve: (tframe, box, h, rho, counts, phi, field, wake)."""
    xl = CLIGHT / (2 * math.pi * c["freq"])
    xt, yt, zt, rcp, bet2 = _tframe(p, gam, xl)
    lo = [min(float((p[0] * xl).min()), float(xt.min())), min(float((p[2] * xl).min()), float(yt.min())),
          float(zt.min())]
    hi = [max(float((p[0] * xl).max()), float(xt.max())), max(float((p[2] * xl).max()), float(yt.max())),
          float(zt.max())]
    box, h = _box(lo, hi, grid)
    i, w = _cic((xt, yt, zt), box, h)
    rho = _deposit(i, w, grid, c["weight"])
    phi = _potential(rho, grid, h)
    e = _field(phi, h)
    wake = None
    if table is not None:
        wake = _wake_planes(c, gam, cur, xt.numel(), xt, yt, zt, box, grid[2], table)
    return dict(t=(xt, yt, zt, rcp, bet2), lo=lo, hi=hi, box=box, h=h, cell=i, rho=rho, phi=phi, e=e,
                wake=wake)


def _gather(p, s, grid, gam, xl):
    """cvbkforth and the field at the particles: (z frame x, y, phase, E, plane weights)."""
    xt, yt, zt, rcp, bet2 = s["t"]
    bi = bet2.sqrt()
    ph1 = zt / xl / (-(gam * bi))
    xg, yg = xt + p[1] * ph1 * rcp * xl, yt + p[3] * ph1 * rcp * xl
    zg = -(gam * bi * ph1 * xl)
    i, w = _cic((xg, yg, zg), s["box"], s["h"])
    i = [k.clamp(0, grid[d] - 2) for d, k in enumerate(i)]
    f = [torch.zeros_like(xg) for _ in range(3)]
    for a, b, cc in CORNERS:
        node, wt = _corner(i, w, grid, a, b, cc)
        for q in range(3):
            f[q] += wt * s["e"][q][node]
    return xg / xl, yg / xl, zg / xl / (-(gam * bi)), f, i[2], w[2]


def _kick(p, s, c, grid, gam, cur, tau, grad, integrator):
    xl = CLIGHT / (2 * math.pi * c["freq"])
    x, y, ph, f, kz, wz = _gather(p, s, grid, gam, xl)
    f = [f[0] * gam, f[1] * gam, f[2]]
    wk = [0.0, 0.0, 0.0]
    if s["wake"] is not None:
        wk = [q[kz] * wz + q[kz + 1] * (1 - wz) for q in s["wake"]]
    if integrator == 2:
        return _lorentz([x, p[1], y, p[3], ph, p[5]], f, gam, tau, xl, c, grad, wk, c["qm"])
    xy, tc = _kick_consts(c, gam, cur)
    if s["wake"] is not None:
        # the map integrator adds the wake to the node fields; a plane's value is the same at
        # all its nodes, so the gather gives its interpolation along z
        q = c["charge"] / c["mass"] / xy / math.sqrt(gam * gam - 1.0)
        f = [f[0] + wk[0] * q * gam, f[1] + wk[1] * q * gam, f[2] + wk[2] * c["charge"] / c["mass"] / tc]
    return [x, p[1] + tau * xy * f[0], y, p[3] + tau * xy * f[1], ph, p[5] - tau * tc * f[2]]


def _exact_run(c, grid, lattice, integrator, table):
    p = [c["pts"][:, k].clone() for k in range(6)]
    gam, cur = -c["ref"][5], c["current"]
    xl = CLIGHT / (2 * math.pi * c["freq"])
    n = float(p[0].numel())
    qm0 = c["charge"] / c["mass"]
    brho = math.sqrt(gam * gam - 1.0) / CLIGHT / qm0
    recs, zs, z = [_record(p, n, cur)], [0.0], 0.0
    for t, length, nseg, _, vals in lattice:
        tau = 0.5 * length / nseg
        if t == 4:
            h0 = vals[0] / length
            p = _pole(p, gam, xl, (h0, "in"), qm0, c["qm"])
            half = lambda q: _sector(q, gam, xl, h0, tau, qm0, c["qm"])  # noqa: E731
        elif integrator == 2:
            half = lambda q: _drift2(q, gam, 2 * tau, xl)  # noqa: E731
        elif t == 0:
            half = lambda q: _drift(q, gam, tau, xl)  # noqa: E731
        elif vals[1] < 0:
            half = lambda q: _kquad(q, gam, tau, xl, vals[0], c["qm"] / qm0)  # noqa: E731
        else:
            half = lambda q: _quad(q, gam, tau, xl, vals[0] / brho)  # noqa: E731
        grad = vals[0] if t == 1 else 0.0
        for _ in range(nseg):
            p = half(p)
            s = _solve(p, c, grid, gam, cur, table)
            p = _kick(p, s, c, grid, gam, cur, 2 * tau, grad, integrator)
            del s
            p = half(p)
            z += tau
            z += tau
            recs.append(_record(p, n, cur))
            zs.append(z)
        if t == 4:
            p = _pole(p, gam, xl, (h0, "out"), qm0, c["qm"])
    return np.array(recs), np.array(zs), p


def _exact_beam(case, m):
    c = _beam(case["beam"], m["n"], m["seed"], m["current"])
    c["weight"], c["qm"] = c["pts"][:, 7].clone(), c["pts"][:, 6].clone()
    return c


def exact(case, seed):
    mem = _members(case, seed)
    if case["kind"] == "static":
        c = _exact_beam(case, mem[0])
        grid = mem[0]["grid"]
        box = _static_box(c, grid).tolist()
        h = [(box[2 * d + 1] - box[2 * d]) / (grid[d] - 1) for d in range(3)]
        xl = CLIGHT / (2 * math.pi * c["freq"])
        t = _tframe([c["pts"][:, k] for k in range(6)], -c["ref"][5], xl)
        i, w = _cic(t[:3], box, h)
        return _deposit(i, w, grid, c["weight"]).view(grid[2], grid[1], grid[0])
    if case["kind"] == "step":
        return _exact_step(case, mem[0])
    table = _wake_table() if case["wake"] else None
    recs, out = [], {}
    for m in mem:
        c = _exact_beam(case, m)
        r, zs, p = _exact_run(c, m["grid"], _lattice(case, m["steps"], m["gradient"]),
                              case["integrator"], table)
        recs.append(r)
    out = _moments(recs)
    if case["kind"] == "run":
        out["z"] = zs
        if case["dump"]:
            out.update({"phase_space%d" % k: p[k] for k in range(6)})
    return out


def _exact_step(case, m):
    c, grid = _exact_beam(case, m), m["grid"]
    t, length, nseg, _, vals = _lattice(case, m["steps"], m["gradient"])[0]
    gam, cur, tau = -c["ref"][5], c["current"], length / nseg / 2
    xl = CLIGHT / (2 * math.pi * c["freq"])
    p = [c["pts"][:, k].clone() for k in range(6)]
    recs = []
    for _ in range(case["steps"]):
        p = _drift(p, gam, tau, xl)
        s = _solve(p, c, grid, gam, cur, None)
        p = _kick(p, s, c, grid, gam, cur, 2 * tau, 0.0, 1)
        p = _drift(p, gam, tau, xl)
        recs.append(_record(p, float(m["n"]), cur))
    out = _moments([np.array(recs)])
    out.update({"ptrange": np.array([v for d in range(3) for v in (s["lo"][d], s["hi"][d])]),
                "range": np.array(s["box"]), "msize": np.array(s["h"])})
    if case["grids"]:
        node = s["cell"][0] + grid[0] * (s["cell"][1] + grid[1] * s["cell"][2])
        counts = torch.bincount(node, minlength=grid[0] * grid[1] * grid[2]).to(torch.int32)
        out.update({"rho": s["rho"], "counts": counts, "phi": s["phi"].reshape(-1),
                    "e": torch.cat(s["e"])})
    return out
