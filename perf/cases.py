"""Performance cases of the engine: simulations as its users run them, through the public API.

A case is one pass of a program: run a simulation (or several, or a stream of requests) for a
number of time steps and read what it is run for.  Kinds:

single  one handle (Sim).  `restart` resets it before every pass, as a parameter sweep does;
        otherwise a pass continues where the last one ended, from initial fields, as a resumed
        run does.  `upload` also gives it new material arrays in every pass.
batch   several handles of uneven size stepped together (Batch).
serve   requests submitted to a Server, waited for and read.

The sizes come from the repository's configurations (512^2 planar, 256^3 drop-in, 512x512x128
photonic-crystal guide, lens batch of sides 128-1024, served cubes of side 64-256, the 34x30x36
smoke grid) and from odd, ragged grids between and beyond them; precision is FP64, FP32 or FP16
storage (prec 0, 1, 2).  `exact` computes the same runs with plain torch operations in 64 bits.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import luxum_gb300 as lx

COMP = ("Ex", "Ey", "Ez", "Hx", "Hy", "Hz")
CELL = 1e-3
EPS0 = 8.85 * pow(10, -12)
MU0 = math.pi * 4 * pow(10, -7)
SIGMA_PW = pow(10, -4) / 0.5
# 0.5-10 GHz, the band of the served requests' flux monitors
BAND = (2 * math.pi * 0.5e9, 2 * math.pi * 10e9)


def listed():
    return [
        # the smallest call: a few dozen steps of a smoke-sized grid, every field read back
        dict(name="tiny_3d_fp64", kind="single", planar=0, nx=34, ny=30, nz=36, prec=0, steps=40, pml=6, wave="x",
             source="none", uniform=1, monitor=0, boxes=1, dft=0, probes=0, series=0, restart=1, upload=0, out="all"),
        # the 512^2 planar configuration: CPML 20, TF/SF plane wave, dielectric box, max|E|^2 of every step
        dict(name="planar_512_fp64", kind="single", planar=1, nx=512, ny=1, nz=512, prec=0, steps=300, pml=20, wave="x",
             source="none", uniform=1, monitor=1, boxes=1, dft=0, probes=0, series=1, restart=1, upload=0, out="all"),
        # a ragged planar grid at an oblique angle, FP32, with a flux monitor
        dict(name="planar_ragged_fp32", kind="single", planar=1, nx=777, ny=1, nz=1031, prec=1, steps=300, pml=16,
             wave="oblique", source="none", uniform=1, monitor=0, boxes=4, dft=32, probes=4, series=0, restart=0, upload=0,
             out="Ey"),
        # a large planar grid
        dict(name="planar_4096_fp32", kind="single", planar=1, nx=4096, ny=1, nz=4096, prec=1, steps=400, pml=20, wave="z",
             source="none", uniform=1, monitor=0, boxes=6, dft=0, probes=4, series=0, restart=0, upload=0, out="Ey"),
        # the 256^3 drop-in run (FP64, CPML 16, TF/SF, probes and max|E|^2 every step), with fields all over the grid
        dict(name="dropin_256_fp64", kind="single", planar=0, nx=256, ny=256, nz=256, prec=0, steps=100, pml=16, wave="x",
             source="none", uniform=1, monitor=1, boxes=1, dft=0, probes=8, series=1, restart=0, upload=0, out="Ez"),
        # a ragged FP64 grid with unequal spacing and an oblique wave, new material uploaded for every run and all
        # fields read: the sweep of a design program
        dict(name="sweep_ragged_fp64", kind="single", planar=0, nx=131, ny=117, nz=150, prec=0, steps=150, pml=9,
             wave="oblique", source="none", uniform=0, monitor=0, boxes=3, dft=0, probes=0, series=0, restart=1, upload=1,
             out="all"),
        # the photonic-crystal guide's grid in FP32: pulsed point source, two FP64 flux planes of 64 frequencies
        dict(name="guide_512x512x128_fp32", kind="single", planar=0, nx=512, ny=512, nz=128, prec=1, steps=200, pml=20,
             wave="none", source="pulse", uniform=1, monitor=0, boxes=40, dft=64, probes=2, series=0, restart=0, upload=0,
             out="Ez"),
        # FP16 storage on an odd grid
        dict(name="odd_3d_fp16", kind="single", planar=0, nx=201, ny=187, nz=259, prec=2, steps=150, pml=12, wave="y",
             source="none", uniform=1, monitor=10, boxes=4, dft=0, probes=4, series=1, restart=0, upload=0, out="Ex"),
        # a small closed cavity with a hard source, read by probes only: launches and nothing else
        dict(name="cavity_64_fp32", kind="single", planar=0, nx=67, ny=64, nz=61, prec=1, steps=200, pml=0, wave="none",
             source="cw", uniform=1, monitor=0, boxes=2, dft=0, probes=6, series=0, restart=0, upload=0, out="Ez"),
        # planar lenses of uneven size as one batch
        dict(name="lens_batch_fp32", kind="batch", planar=1, count=48, lo=128, hi=1024, prec=1, steps=300, pml=16, dft=0),
        # 3-D requests' cubes as one batch, each with a flux plane
        dict(name="cube_batch_fp32", kind="batch", planar=0, count=10, lo=48, hi=176, prec=1, steps=200, pml=12, dft=16),
        # a burst of requests through the server, planar and 3-D
        dict(name="serve_burst_fp32", kind="serve", count=32, prec=1, steps=400, chunk=100),
    ]


def draw(rng):
    def logint(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    kind = rng.choice(["single", "single", "single", "single", "batch", "serve"])
    prec = rng.choice([0, 1, 1, 2])
    if kind == "serve":
        return dict(kind="serve", count=rng.randint(4, 32), prec=1, steps=rng.choice([150, 300, 400]),
                    chunk=rng.choice([50, 100]))
    planar = rng.choice([0, 1])
    if kind == "batch":
        if planar:
            return dict(kind="batch", planar=1, count=rng.randint(4, 48), lo=128, hi=logint(256, 1024), prec=prec,
                        steps=rng.randint(100, 300), pml=rng.randint(6, 16), dft=rng.choice([0, 16]))
        return dict(kind="batch", planar=0, count=rng.randint(2, 10), lo=32, hi=logint(64, 176), prec=prec,
                    steps=rng.randint(50, 200), pml=rng.randint(5, 12), dft=rng.choice([0, 16]))
    c = dict(kind="single", planar=planar, prec=prec)
    if planar:
        c.update(nx=logint(64, 4096), ny=1, nz=logint(64, 4096))
        cells, cap = c["nx"] * c["nz"], 6e9
    else:
        c.update(nx=logint(26, 400), ny=logint(26, 300), nz=logint(26, 400))
        cells, cap = c["nx"] * c["ny"] * c["nz"], 1.6e9
    c["steps"] = max(20, min(rng.randint(40, 300), int(cap / cells)))
    side = min(c["nx"], c["nz"]) if planar else min(c["nx"], c["ny"], c["nz"])
    c["pml"] = rng.choice([0, 1, 1]) * rng.randint(5, max(5, min(20, side // 6)))
    c["wave"] = rng.choice(["x", "z", "oblique"] if planar else ["x", "y", "z", "oblique"])
    c["source"] = "none"
    if rng.random() < 0.25:
        c["wave"], c["source"] = "none", "pulse"
    c["uniform"] = rng.choice([0, 1, 1])
    c["monitor"] = rng.choice([0, 1, 10])
    c["boxes"] = rng.randint(1, 6)
    c["restart"] = rng.choice([0, 1])
    # a run from zero fields is too short for the wave to be at the flux planes, and fills its own component first
    c["dft"] = 0 if c["restart"] else rng.choice([0, 16, 64])
    c["probes"] = 0 if c["restart"] else rng.choice([0, 4, 8])
    c["series"] = 1 if c["monitor"] else 0
    c["upload"] = 0
    main = {"x": "Ez", "y": "Ex", "z": "Ey", "oblique": "Ex", "none": "Ez"}[c["wave"]]
    c["out"] = "Ey" if planar else main if c["restart"] else rng.choice(COMP)
    return c


# ---------------------------------------------------------------------- what a program sets up


def _spacing(case):
    if case.get("uniform", 1):
        return CELL, CELL, CELL
    return CELL, 1.25 * CELL, 0.9 * CELL


def _wave(kind, planar):
    if kind == "x":
        return (1.0, 0.0, 0.0), ((0.0, 1.0, 0.0) if planar else (0.0, 0.0, 1.0))
    if kind == "y":
        return (0.0, 1.0, 0.0), (1.0, 0.0, 0.0)
    if kind == "z":
        return (0.0, 0.0, 1.0), (0.0, 1.0, 0.0)
    if planar:
        return (0.6, 0.0, 0.8), (0.0, 1.0, 0.0)
    s3, s2 = 1 / math.sqrt(3), 1 / math.sqrt(2)
    return (s3, s3, s3), (s2, 0.0, -s2)


def _keywords(n, planar, prec, steps, pml, wave, spacing, monitor, source="none", src=None):
    """Keyword arguments of lx.params for one simulation."""
    dx, dy, dz = spacing
    kw = dict(isPlanar=planar, Nx=n[0], Ny=n[1], Nz=n[2], dx=dx, dy=dy, dz=dz, S=0.5, num_timesteps=steps, precision=prec,
              monitor_every=monitor)
    if pml:
        kw.update(usePML=1, d_pml=pml * max(dx, dz, 0.0 if planar else dy), sigma=0.65, sigma_m=3.0, kappa=5.0, a_max=0.05,
                  a_m=1.0, cpml_mode=lx.LX_CPML_STANDARD)
    if wave != "none":
        k, e = _wave(wave, planar)
        lo = [0 if (planar and a == 1) else max(2, int(1.5 * pml) + 2) for a in range(3)]
        hi = [n[a] - 1 - lo[a] for a in range(3)]
        front = sum(lo[a] * d * k[a] for a, d in enumerate(spacing)) / dx
        # the pulse (14 cells at 1/e) starts 30 cells before the box
        kw.update(usePW=1, kx_pw=k[0], ky_pw=k[1], kz_pw=k[2], Ex_pw=e[0], Ey_pw=e[1], Ez_pw=e[2], off_pw=30.0 - front,
                  x1_pw=lo[0], x2_pw=hi[0], y1_pw=lo[1], y2_pw=hi[1], z1_pw=lo[2], z2_pw=hi[2])
    if source != "none":
        kw.update(usePS=1, Nx_source=src[0], Ny_source=src[1], Nz_source=src[2])
        if source == "cw":
            kw.update(source_kind=lx.LX_SRC_CW_HARD, amp_source=400.0, omega_source=1.0e9)
        else:
            kw.update(source_kind=lx.LX_SRC_PULSE_SOFT, amp_source=1.0, omega_source=2 * math.pi * 5e9, src_t0=60.0,
                      src_tw=25.0)
    return kw


def _boxes(rng, n, planar, count, margin):
    got = []
    for _ in range(count):
        lo, hi = [], []
        for a in range(3):
            if planar and a == 1:
                lo.append(0)
                hi.append(1)
                continue
            w = int(rng.integers(3, max(4, n[a] // 6)))
            first, last = margin + 1, max(margin + 2, n[a] - margin - 1 - w)
            s = int(rng.integers(first, last))
            lo.append(s)
            hi.append(s + w)
        got.append((tuple(lo), tuple(hi), float(rng.uniform(1.5, 11.0))))
    return got


def _initial(n, planar, seed, shapes):
    """Smooth random E and H, zero at the walls: a few oblique sinusoids under a window."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    rng = np.random.default_rng(seed + 77)
    ax = [torch.arange(m, dtype=torch.float64, device=dev) for m in n]
    win = [torch.sin(math.pi * a / max(m - 1, 1)) if m > 1 else torch.ones(1, dtype=torch.float64, device=dev)
           for a, m in zip(ax, n)]
    win = win[0][:, None, None] * win[1][None, :, None] * win[2][None, None, :]
    out = []
    for c in range(6):
        scale = 1.0 if c < 3 else 1.0 / 377.0
        if 0 in shapes[c]:
            out.append(None)
            continue
        k = rng.uniform(0.05, 0.5, 3)
        ph = rng.uniform(0, 2 * math.pi, 3)
        f = (torch.sin(k[0] * ax[0] + ph[0])[:, None, None] + torch.sin(k[1] * ax[1] + ph[1])[None, :, None]) * torch.cos(
            k[2] * ax[2] + ph[2])[None, None, :] * win * (scale * (0.5 + rng.random()))
        s = shapes[c]
        out.append(f[: s[0], : s[1], : s[2]].contiguous().cpu().numpy())
    return out


def _single(case, seed):
    """Everything about a single run but its handle."""
    rng = np.random.default_rng(seed)
    planar = case["planar"]
    n = (case["nx"], case["ny"], case["nz"])
    mid = [int(m // 2 + rng.integers(-m // 8, m // 8 + 1)) if m > 1 else 0 for m in n]
    kw = _keywords(n, planar, case["prec"], case["steps"], case["pml"], case["wave"], _spacing(case), case["monitor"],
                   case["source"], mid)
    margin = int(1.5 * case["pml"]) + 2
    boxes = _boxes(rng, n, planar, case["boxes"], margin)
    probes = [[int(rng.integers(1, m - 1)) if m > 1 else 0 for m in n] for _ in range(case["probes"])]
    planes = []
    if case["dft"]:
        omega = np.linspace(BAND[0], BAND[1], case["dft"])
        planes = [(0, n[0] // 4, omega, 5), (0, n[0] - 1 - n[0] // 4, omega, 5)]
    return dict(kw=kw, n=n, planar=planar, boxes=boxes, probes=probes, planes=planes)


def _material(d, shape):
    """F of the material form Cb = dt/(eps0*(1+F)) for the boxes."""
    F = np.zeros(shape)
    for lo, hi, eps in d["boxes"]:
        F[lo[0]:hi[0], lo[1]:hi[1], lo[2]:hi[2]] = eps - 1.0
    return F


def _members(case, seed):
    """Parameters, boxes and flux plane of each member of a batch, or each request of a stream.
    The sizes are the case's, what stands in the grids is the seed's."""
    rng, sizes = np.random.default_rng(seed), np.random.default_rng(1000 + case["count"])
    got = []
    for q in range(case["count"]):
        pick = sizes.random()
        planar = case.get("planar", 0 if pick < 0.2 else 1)
        lo, hi = (case["lo"], case["hi"]) if "lo" in case else ((200, 1024) if planar else (48, 128))
        side = int(round(math.exp(sizes.uniform(math.log(lo), math.log(hi)))))
        if "lo" in case:  # the ends of the range are always there
            side = lo if q == 0 else hi if q == 1 else side
        m = min(case.get("pml", 16), side // 8)
        n = (side, 1 if planar else side, side + int(sizes.integers(0, 9)))
        kw = _keywords(n, planar, case["prec"], case["steps"], m, "x", (CELL, CELL, CELL), 0)
        plane = None
        if case.get("dft", 16):
            plane = (0, 2 * m + 12, np.linspace(BAND[0], BAND[1], case.get("dft", 16)), 10)
        got.append(dict(kw=kw, n=n, planar=planar, boxes=_boxes(rng, n, planar, int(rng.integers(1, 5)), 2 * m + 2),
                        plane=plane))
    return got


def prepare(case, seed):
    if case["kind"] == "single":
        d = _single(case, seed)
        sim = lx.Sim(lx.params(**d["kw"]))
        names = COMP if case["out"] == "all" else (case["out"],)
        state = dict(case=case, sim=sim, d=d, outs=[COMP.index(c) for c in names if np.prod(sim.shape(COMP.index(c)))])
        if case["upload"]:
            state["F"] = [_material(d, sim.shape(c)) for c in range(3)]
        else:
            for lo, hi, eps in d["boxes"]:
                sim.set_eps_box(lo, hi, eps)
        if not case["restart"]:
            for c, f in enumerate(_initial(d["n"], d["planar"], seed, [sim.shape(c) for c in range(6)])):
                if f is not None:
                    sim.set_field(c, f)
        state["planes"] = [sim.add_dft_plane(*p) for p in d["planes"]]
        if d["probes"]:
            sim.set_probes(d["probes"], case["steps"])
        if case["series"]:
            sim.set_max_series(case["steps"] + 1)
        return state
    members = _members(case, seed)
    if case["kind"] == "serve":
        return dict(case=case, server=lx.Server(precision=case["prec"], chunk=case["chunk"]), members=members)
    batch = lx.Batch(chunk=100)
    sims, planes = [], []
    for m in members:
        s = lx.Sim(lx.params(**m["kw"]))
        for lo, hi, eps in m["boxes"]:
            s.set_eps_box(lo, hi, eps)
        planes.append(s.add_dft_plane(*m["plane"]) if m["plane"] else None)
        batch.add(s)
        sims.append(s)
    return dict(case=case, batch=batch, sims=sims, planes=planes)


def run(state):
    case = state["case"]
    if case["kind"] == "single":
        sim = state["sim"]
        if case["upload"]:
            for c in range(3):
                sim.set_material(c, state["F"][c], 1.0)
        if case["restart"]:
            sim.reset()
        elif state["d"]["probes"]:
            sim.set_probes(state["d"]["probes"], case["steps"])  # a new recording of the steps that follow
        sim.step(case["steps"])
        out = {COMP[c]: sim.field(c) for c in state["outs"]}
        if state["d"]["probes"]:
            out["probes"] = sim.probes()
        if case["series"]:
            out["max_e2"] = sim.max_series()[1]
        for q, p in enumerate(state["planes"]):
            out["flux%d" % q] = sim.dft_flux(p)
        return out
    if case["kind"] == "batch":
        state["batch"].step(case["steps"])
        return [s.field(1 if case["planar"] else 2) if p is None else s.dft_flux(p)
                for s, p in zip(state["sims"], state["planes"])]
    srv = state["server"]
    ids = [srv.submit(lx.params(**m["kw"]), case["steps"], m["boxes"], m["plane"]) for m in state["members"]]
    out = []
    for rid in ids:
        if srv.wait(rid) != "done":
            raise RuntimeError(srv.error(rid))
        out.append(srv.flux(rid))
        srv.release(rid)
    return out


# ---------------------------------------------------------------------- the work of a pass


def _step_work(n, planar, prec, pml, uniform=True):
    """Compulsory bytes of a time step (each field read and written once, the material coefficients read
    once, each psi entry of the absorbing layers read and written once) and its operations."""
    cells = float(n[0] * n[1] * n[2])
    ts, cs = (8, 4, 2)[prec], (8, 4, 4)[prec]
    b = cells * (2 * (3 if planar else 6) * ts + (1 if planar else 3) * cs)
    f = cells * (4 + 4 + 4 if planar else 30)
    if pml:
        for a in range(3):
            if planar and a == 1:
                continue
            psi = min(2 * pml, n[a]) * cells / n[a] * (2 if planar else 4)
            b += 2 * psi * cs
            f += 5 * psi
    return b, f


def work(case):
    if case["kind"] == "single":
        n = (case["nx"], case["ny"], case["nz"])
        b, f = _step_work(n, case["planar"], case["prec"], case["pml"])
        outs = (3 if case["planar"] else 6) if case["out"] == "all" else 1
        cells = float(n[0] * n[1] * n[2])
        dft = 2.0 * case["dft"] * 4 * n[1] * n[2] * ((case["steps"] + 4) // 5)
        return {"bytes": b * case["steps"] + 8 * cells * (outs + (3 if case["upload"] else 0)) + 32 * dft,
                "flops": f * case["steps"] + 4 * dft}
    total = {"bytes": 0.0, "flops": 0.0}
    for m in _members(case, 0):
        b, f = _step_work(m["n"], m["planar"], case["prec"], min(case.get("pml", 16), m["n"][0] // 8))
        total["bytes"] += b * case["steps"]
        total["flops"] += f * case["steps"]
        if m["plane"]:
            dft = len(m["plane"][2]) * 4.0 * m["n"][1] * m["n"][2] * ((case["steps"] + 9) // 10)
            total["bytes"] += 32 * dft
            total["flops"] += 4 * dft
        elif case["kind"] == "batch":
            total["bytes"] += 8.0 * m["n"][0] * m["n"][1] * m["n"][2]
    return total


# ---------------------------------------------------------------------- the same runs in plain 64-bit torch


def _profiles(N, delta, kw, dt):
    """kappa, b, c at the E (integer) and H (half) positions of one axis, as the solver defines them."""
    got = []
    d = kw["d_pml"] / delta
    s_max = 0.8 * (kw["sigma_m"] + 1) / kw["dx"] / math.sqrt(MU0 / EPS0) * kw["sigma"]
    for half, m in ((0.0, N), (0.5, N - 1)):
        t = np.arange(m) + half
        depth = np.where(t <= d - 1, (d - 1 - t) / (d - 1), np.where(t >= N - d, (t - N + d) / (d - 1), 0.0))
        inside = (t <= d - 1) | (t >= N - d)
        sg = np.where(inside, depth ** kw["sigma_m"] * s_max, 0.0)
        ka = np.where(inside, depth ** kw["sigma_m"] * (kw["kappa"] - 1) + 1, 1.0)
        aa = np.where(t <= d - 1, (t / (d - 1)) ** kw["a_m"] * kw["a_max"], 0.0)
        back = np.where(t >= N - d, np.maximum(N - 1 - t, 0.0) / (d - 1), 0.0)
        aa = np.where(t >= N - d, back ** kw["a_m"] * kw["a_max"], aa)
        b = np.exp(-(sg / ka / EPS0 + aa / EPS0) * dt)
        den = sg * ka + ka ** 2 * aa
        c = np.where(sg == 0, 0.0, sg / np.where(den == 0, 1.0, den) * (b - 1))
        got.append((ka, b, c))
    return got


class _Exact:
    """The Yee scheme with CPML, TF/SF plane wave, point source and DFT planes, whole arrays at a time."""

    def __init__(self, kw, boxes, init=None):
        self.kw, self.planar = kw, kw["isPlanar"]
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.n = n = (kw["Nx"], kw["Ny"], kw["Nz"])
        self.sp = (kw["dx"], kw["dy"], kw["dz"])
        self.c = 1 / math.sqrt(EPS0 * MU0)
        self.dt = kw["S"] * kw["dx"] / self.c
        z = lambda: torch.zeros(n, dtype=torch.float64, device=self.dev)  # noqa: E731
        self.F = [z() for _ in range(6)]
        for c, f in enumerate(init or []):
            if f is not None:
                s = f.shape
                self.F[c][: s[0], : s[1], : s[2]] = torch.from_numpy(f).to(self.dev)
        eps = torch.ones(n, dtype=torch.float64, device=self.dev)
        for lo, hi, e in boxes:
            eps[lo[0]:hi[0], lo[1]:hi[1], lo[2]:hi[2]] = e
        self.Cb = self.dt / (EPS0 * eps)
        self.Db = self.dt / MU0
        N = [n[0], n[1], n[2]]
        last = [m - 1 for m in N]
        full = [slice(0, m) for m in N]
        up = [slice(0, m - 1) for m in N]
        mid = [slice(1, m - 1) for m in N]
        # component -> (region, [(axis, source component, sign)] of its two curl parts)
        if self.planar:
            self.hreg = {0: (full[0], full[1], up[2]), 2: (up[0], full[1], full[2])}
            self.hparts = {0: [(2, 1, -1.0)], 2: [(0, 1, +1.0)]}
            self.ereg = {1: (mid[0], full[1], mid[2])}
            self.eparts = {1: [(2, 3, +1.0), (0, 5, -1.0)]}
        else:
            self.hreg = {0: (full[0], up[1], up[2]), 1: (up[0], full[1], up[2]), 2: (up[0], up[1], full[2])}
            self.hparts = {0: [(1, 2, +1.0), (2, 1, -1.0)], 1: [(2, 0, +1.0), (0, 2, -1.0)], 2: [(0, 1, +1.0), (1, 0, -1.0)]}
            self.ereg = {0: (up[0], mid[1], mid[2]), 1: (mid[0], up[1], mid[2]), 2: (mid[0], mid[1], up[2])}
            self.eparts = {0: [(1, 5, +1.0), (2, 4, -1.0)], 1: [(2, 3, +1.0), (0, 5, -1.0)], 2: [(0, 4, +1.0), (1, 3, -1.0)]}
        self.last = last
        self.prof, self.psi = {}, {}
        if kw.get("usePML"):
            for a in range(3):
                if self.planar and a == 1:
                    continue
                for h, (ka, b, c) in zip("EH", _profiles(n[a], self.sp[a], kw, self.dt)):
                    shape = [1, 1, 1]
                    shape[a] = -1
                    pad = n[a] - len(ka)
                    self.prof[h, a] = [torch.from_numpy(np.concatenate([v, np.full(pad, fill)])).to(self.dev).reshape(shape)
                                       for v, fill in ((ka, 1.0), (b, 1.0), (c, 0.0))]
        self.sets = self._sets() if kw.get("usePW") else []
        self.t = 0

    def _sets(self):
        """(for E, component, axis, plane, sign, position, in-plane ranges, offsets, factor) of each TF/SF plane."""
        kw = self.kw
        k = np.array([kw["kx_pw"], kw["ky_pw"], kw["kz_pw"]])
        E = np.array([kw["Ex_pw"], kw["Ey_pw"], kw["Ez_pw"]])
        H = np.cross(k, E)
        H = H / np.linalg.norm(H)
        lo = [kw["x1_pw"], kw["y1_pw"], kw["z1_pw"]]
        hi = [kw["x2_pw"], kw["y2_pw"], kw["z2_pw"]]
        if self.planar:
            lo[1] = hi[1] = 0
        stag = {0: (0.5, 0, 0), 1: (0, 0.5, 0), 2: (0, 0, 0.5)}  # the wave's E component c, and H component c's source
        got = []
        for isE, parts in ((0, self.hparts), (1, self.eparts)):
            for comp, ps in parts.items():
                for axis, src, _ in ps:
                    amp = E[src] if not isE else H[src - 3]
                    if amp == 0.0:
                        continue
                    sgn = -1.0 if self.planar else 1.0  # the planar lines inject the wave with amplitude -1
                    # in-plane staggering: that of the E component on the plane (the source for H, the target for E)
                    e_comp = src if not isE else comp
                    off = [0.0 if (self.planar and a == 1) else stag[e_comp][a] for a in range(3)]
                    f = sgn * amp / self.sp[axis]
                    if isE:
                        f = f / self.c / MU0
                    for q in (0, 1):
                        if not isE:
                            plane, pos = (lo[axis] - 1, lo[axis]) if q == 0 else (hi[axis], hi[axis])
                        else:
                            plane, pos = (lo[axis], lo[axis] - 0.5) if q == 0 else (hi[axis], hi[axis] + 0.5)
                        sign = -1.0 if q == 0 else 1.0
                        rng = [(lo[a], hi[a] - (1 if off[a] else 0)) for a in range(3)]
                        got.append((isE, comp, axis, plane, sign, pos, rng, off, f))
        return got

    def _incident(self, isE, comp, axis, d, reg):
        kw = self.kw
        for sE, c, a, plane, sign, pos, rng, off, f in self.sets:
            if sE != isE or c != comp or a != axis:
                continue
            X = torch.zeros((1, 1, 1), dtype=torch.float64, device=self.dev)
            idx = []
            for b, kb in enumerate((kw["kx_pw"], kw["ky_pw"], kw["kz_pw"])):
                if b == a:
                    p = torch.tensor([float(pos)], dtype=torch.float64, device=self.dev)
                    idx.append(slice(plane - reg[b].start, plane - reg[b].start + 1))
                else:
                    p = torch.arange(rng[b][0], rng[b][1] + 1, dtype=torch.float64, device=self.dev) + off[b]
                    idx.append(slice(rng[b][0] - reg[b].start, rng[b][1] + 1 - reg[b].start))
                if self.planar and b == 1:
                    continue
                s = [1, 1, 1]
                s[b] = -1
                X = X + (p * self.sp[b] * kb).reshape(s)
            tt = self.t if isE else self.t - 0.5
            X = X + kw["off_pw"] * self.sp[0] - tt * self.c * self.dt
            v = torch.exp(-X * X / SIGMA_PW) * f
            d[tuple(idx)] += sign * v
        return d

    def _curl(self, isE, comp, axis, src, reg):
        A = self.F[src]
        # the neighbour difference along axis over the region: forward for H, backward for E
        lo, hi = list(reg), list(reg)
        if isE:
            lo[axis] = slice(reg[axis].start - 1, reg[axis].stop - 1)
        else:
            hi[axis] = slice(reg[axis].start + 1, reg[axis].stop + 1)
        d = (A[tuple(hi)] - A[tuple(lo)]) / self.sp[axis]
        d = self._incident(isE, comp, axis, d, reg)
        if ("E" if isE else "H", axis) in self.prof:
            ka, b, c = [v[tuple(reg[x] if x == axis else slice(0, 1) for x in range(3))] for v in
                        self.prof["E" if isE else "H", axis]]
            key = (isE, comp, axis)
            if key not in self.psi:
                self.psi[key] = torch.zeros_like(d)
            self.psi[key] = b * self.psi[key] + c * d
            d = d / ka + self.psi[key]
        return d

    def step(self):
        kw, t = self.kw, self.t
        if kw.get("usePS"):
            i = (kw["Nx_source"], 0 if self.planar else kw["Ny_source"], kw["Nz_source"])
            if kw["source_kind"] == lx.LX_SRC_CW_HARD:
                wt = (int(kw["omega_source"]) * t) & 0xFFFFFFFF
                wt = wt - (1 << 32) if wt >= 1 << 31 else wt
                self.F[2][i] = int(kw["amp_source"]) * math.sin(wt * self.dt)
            else:
                u = (t - kw["src_t0"]) / kw["src_tw"]
                self.F[1 if self.planar else 2][i] += kw["amp_source"] * math.exp(-u * u) * math.sin(kw["omega_source"] * t * self.dt)
        for isE, regs, parts in ((0, self.hreg, self.hparts), (1, self.ereg, self.eparts)):
            new = {}
            for comp, reg in regs.items():
                tot = 0.0
                for axis, src, sign in parts[comp]:
                    tot = tot + sign * self._curl(isE, comp, axis, src, reg)
                new[comp] = tot
            for comp, reg in regs.items():
                if isE:
                    self.F[comp][reg] += self.Cb[reg] * new[comp]
                else:
                    self.F[3 + comp][reg] -= self.Db * new[comp]
        self.t += 1

    def max_e2(self):
        if self.planar:
            return float((self.F[1] ** 2).max())
        r = tuple(slice(0, m) for m in self.last)
        return float((self.F[0][r] ** 2 + self.F[1][r] ** 2 + self.F[2][r] ** 2).max())

    def shape(self, c):
        n = self.n
        if self.planar:
            return {1: (n[0], 1, n[2]), 3: (n[0], 1, n[2] - 1), 5: (n[0] - 1, 1, n[2])}.get(c, (0, 0, 0))
        return tuple(n[a] - (1 if (a == c if c < 3 else a != c - 3) else 0) for a in range(3))

    def field(self, c):
        s = self.shape(c)
        return self.F[c][: s[0], : s[1], : s[2]].cpu().numpy()


class _Plane:
    """Running DFT of the tangential fields on an x plane, and its net flux."""

    def __init__(self, ex, plane):
        _, self.index, self.omega, self.every = plane
        self.acc = torch.zeros((4, len(self.omega)) + tuple(ex.n[1:]), dtype=torch.complex128, device=ex.dev)

    def sample(self, ex, t):
        if t % self.every:
            return
        w = torch.from_numpy(np.asarray(self.omega)).to(ex.dev)
        for q, c in enumerate((1, 2, 4, 5)):
            s = ex.shape(c)
            if 0 in s or self.index >= s[0]:
                continue
            v = torch.zeros(ex.n[1:], dtype=torch.float64, device=ex.dev)
            v[: s[1], : s[2]] = ex.F[c][self.index, : s[1], : s[2]]
            ph = w * ((t + (1.0 if c < 3 else 0.5)) * ex.dt)
            self.acc[q] += torch.polar(torch.full_like(ph, float(self.every)), -ph)[:, None, None] * v

    def flux(self, ex):
        a = self.acc
        p = (a[0] * a[3].conj() - a[1] * a[2].conj()).real.sum(dim=(1, 2))
        dA = ex.sp[2] if ex.planar else ex.sp[1] * ex.sp[2]
        return (p * dA).cpu().numpy()


def exact(case, seed):
    if case["kind"] == "single":
        n = (case["nx"], case["ny"], case["nz"])
        d = _single(case, seed)
        ex = _Exact(d["kw"], d["boxes"])
        if not case["restart"]:
            shapes = [ex.shape(c) for c in range(6)]
            ex = _Exact(d["kw"], d["boxes"], _initial(n, d["planar"], seed, shapes))
        planes = [_Plane(ex, p) for p in d["planes"]]
        probes = np.zeros((case["steps"], len(d["probes"]), 6))
        series = []
        for t in range(case["steps"]):
            ex.step()
            for p in planes:
                p.sample(ex, t)
            for q, i in enumerate(d["probes"]):
                for c in range(6):
                    if all(a < b for a, b in zip(i, ex.shape(c))):
                        probes[t, q, c] = ex.F[c][tuple(i)]
            if case["series"] and (t == case["steps"] - 1 or (case["monitor"] and (t + 1) % case["monitor"] == 0)):
                series.append(ex.max_e2())
        names = COMP if case["out"] == "all" else (case["out"],)
        out = {c: ex.field(COMP.index(c)) for c in names if np.prod(ex.shape(COMP.index(c)))}
        if d["probes"]:
            out["probes"] = probes
        if case["series"]:
            out["max_e2"] = np.array(series)
        for q, p in enumerate(planes):
            out["flux%d" % q] = p.flux(ex)
        return out
    out = []
    members = _members(case, seed)
    # seconds a step: the operations' launches on small arrays, the cells on large ones
    if sum(case["steps"] * ((2e-3 if m["planar"] else 5e-3) + 1.2e-9 * np.prod(m["n"])) for m in members) > 15:
        keep = set(range(0, len(members), max(1, len(members) // 8)))
    else:
        keep = set(range(len(members)))
    for q, m in enumerate(members):
        if q not in keep:
            out.append(None)
            continue
        ex = _Exact(m["kw"], m["boxes"])
        plane = _Plane(ex, m["plane"]) if m["plane"] else None
        for t in range(case["steps"]):
            ex.step()
            if plane:
                plane.sample(ex, t)
        out.append(plane.flux(ex) if plane else ex.field(1 if case["planar"] else 2))
    return out
