"""The work that users of this framework have it do, as measurable cases over its public entry points.

A case is one call sequence of a user's program on one kind of problem:
  grid     a time-domain run (TMxll): a stretch of the time loop of a simulation that is under way
           (fields, media, a driving source, optionally quantum emitters), its detector records
           drained and a field snapshot and the emitters read at its end
  sweep    the same for several 3D grids advanced together (Batch), as in a parameter sweep
  solve    the frequency-domain solver of an inverse-design iteration (FDOperator.solve)
  network  the learned emitter closure: its inference on field histories (Closure.forward) or the
           loss and gradient of a training batch (Closure.gradient)
`exact` computes the same results with torch in 64 bits, without the framework.
"""
import math
import os
import random
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))),
                                "one-mxll-to-rule-them-all_gb300"))
import omx  # noqa: E402
from omx.units import UNITS, yee_dt  # noqa: E402

NM, EV, FS, DEBYE = UNITS["nm_to_au"], UNITS["ev_to_au"], UNITS["fs_to_au"], UNITS["Debye_to_au"]
C0, EPS0, MU0 = UNITS["c0"], UNITS["eps0"], UNITS["mu0"]
EX, EY, EZ, HX, HY, HZ = 1, 2, 3, 4, 5, 6
KIND = {"c": omx.CPML, "p": omx.PERIODIC, "w": omx.CLOSE}      # open, periodic, closed walls


# ---- the cases ---------------------------------------------------------------------------------
def _grid(dims, n, mode, prec, bnd, npml, dr_nm, scene, emitters, steps, every, calls=False):
    n = list(n) + [1] * (3 - len(n))
    return dict(kind="grid", dims=dims, nx=n[0], ny=n[1], nz=n[2], mode=mode, prec=prec, bnd=bnd, npml=npml,
                dr_nm=dr_nm, scene=scene, emitters=emitters, steps=steps, every=every, calls=calls)


def listed():
    return [
        # a pulse through a thin film on one axis, in the reference's own precision: the smallest grid
        dict(_grid(1, (1501,), "x", "fp64", "c", 10, 1.0, "drude", 16, 500, 1), name="film_1d_fp64"),
        # a small TMz scene under a host program that keeps the reference's loop, one call per step part
        dict(_grid(2, (243, 161), "tmz", "fp32", "pc", 8, 2.0, "drude", 300, 100, 1, True), name="tmz_calls_243x161"),
        # the 2D flagship: a perforated silver film, 1e4 emitters, the loop on the device
        dict(_grid(2, (4096, 4096), "tmz", "fp32", "pc", 10, 2.0, "drude", 10000, 400, 10), name="tmz_4096"),
        # the other 2D polarisation, a pixelated dielectric design on a ragged grid
        dict(_grid(2, (1531, 1147), "tez", "fp32", "cc", 10, 10.0, "pixels", 0, 200, 4), name="tez_1531x1147"),
        # a dispersive sphere with molecules in the reference's own precision: the bit-parity path
        dict(_grid(3, (88, 76, 67), "full", "fp64", "ccc", 8, 2.0, "gold", 2000, 100, 1), name="sphere_3d_fp64"),
        # the plain 3D configuration: gold nanosphere, 128^3
        dict(_grid(3, (128, 128, 128), "full", "fp32", "ccc", 10, 2.0, "gold", 0, 400, 1), name="sphere_128"),
        # a metasurface unit cell: periodic in the plane, open along z
        dict(_grid(3, (101, 90, 157), "full", "fp32", "ppc", 10, 5.0, "pixels", 0, 200, 4), name="unit_cell_101x90x157"),
        # a large plasmonic scene with 1e5 three-level molecules
        dict(_grid(3, (320, 288, 250), "full", "fp32", "ccc", 10, 1.0, "gold", 100000, 60, 1), name="dimers_320x288x250"),
        # an inverse-design sweep: twelve small dielectric grids advanced together
        dict(kind="sweep", count=12, lo=48, hi=112, npml=8, dr_nm=20.0, steps=100, every=4, sides=12,
             name="sweep_12_grids"),
        # the field solve of one design iteration
        dict(kind="solve", dims=3, nx=30, ny=27, nz=25, npml=6, nder=2, bnd="ccc", L=2, tol=1e-6, name="solve_30x27x25"),
        # the emitter network on the field histories of a group of molecules
        dict(kind="network", what="forward", rows=20000, T=32, skip=0, name="network_forward_20000"),
        # one training batch of whole trajectories (160 samples)
        dict(kind="network", what="gradient", rows=256, T=129, skip=4, name="network_gradient_256"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    k = rng.choice(["1d", "tmz", "tez", "fp64", "3d", "3d", "cell", "sweep", "solve", "forward", "gradient"])
    every = rng.choice([1, 2, 5])
    if k == "1d":
        return _grid(1, (_log(rng, 200, 8000),), "x", rng.choice(["fp64", "fp32"]), "c", rng.choice([8, 10, 12]), 1.0,
                     rng.choice(["drude", "pixels"]), rng.choice([0, 8, 33]), _log(rng, 100, 600), every)
    if k in ("tmz", "tez"):
        n = (_log(rng, 100, 4000), _log(rng, 90, 4000))
        return _grid(2, n, k, "fp32", rng.choice(["pc", "cc"]), rng.choice([8, 10]), 2.0,
                     rng.choice(["drude", "pixels"]), rng.choice([0, min(n[0], 2000)]),
                     min(200, max(20, int(4e8 / (n[0] * n[1])))), 5 * every, n[0] * n[1] < 1e5 and rng.random() < 0.5)
    if k == "fp64":
        return _grid(3, [_log(rng, 24, 128) for _ in range(3)], "full", "fp64", rng.choice(["ccc", "ppc"]), 6, 2.0,
                     rng.choice(["gold", "pixels"]), rng.choice([0, 400]), 50, every)
    if k in ("3d", "cell"):
        n = [_log(rng, 32, 288) for _ in range(3)]
        return _grid(3, n, "full", "fp32", "ccc" if k == "3d" else rng.choice(["ppc", "pcc", "ppp"]),
                     rng.choice([6, 8, 10]), 2.0, rng.choice(["gold", "pixels"]), rng.choice([0, 500]),
                     min(200, max(20, int(6e8 / (n[0] * n[1] * n[2])))), every)
    if k == "sweep":
        return dict(kind="sweep", count=rng.randint(3, 16), lo=rng.randint(28, 48), hi=rng.randint(56, 112), npml=6,
                    dr_nm=20.0, steps=rng.randint(20, 80), every=4, sides=rng.randint(1, 9999))
    if k == "solve":
        two = rng.random() < 0.5
        n = [_log(rng, 40, 90), _log(rng, 40, 90), 1] if two else [_log(rng, 20, 32) for _ in range(3)]
        return dict(kind="solve", dims=2 if two else 3, nx=n[0], ny=n[1], nz=n[2], npml=5, nder=rng.choice([1, 2, 3]),
                    bnd="cc" if two else rng.choice(["ccc", "pcc"]), L=rng.choice([1, 2, 4]), tol=1e-6)
    if k == "forward":
        return dict(kind="network", what="forward", rows=8 * _log(rng, 8, 4000), T=_log(rng, 4, 40), skip=0)
    return dict(kind="network", what="gradient", rows=8 * _log(rng, 8, 128), T=_log(rng, 8, 129), skip=4)


# ---- inputs from the seed, the same for the framework and for `exact` ----------------------------
MEDIA = {
    "drude": dict(kind="drude", wp=9.17, gamma=0.021, eps=1.0),                       # silver
    "gold": dict(kind="dl", wp=9.0, gamma=0.07, eps=5.9, poles=[2.7, 3.9], strengths=[1.0, 0.6], widths=[0.3, 0.5]),
    "pixels": dict(kind="dielectric", eps=12.1),
}


def _scene(c, seed):
    """A grid case's inputs: medium mask, initial fields, source, emitters, detectors."""
    rng = np.random.default_rng([seed, c["nx"], c["ny"], c["nz"], c["steps"]])
    d, npml = c["dims"], c["npml"]
    n = [c["nx"], c["ny"], c["nz"]][:d]
    dr = c["dr_nm"] * NM
    s = dict(n=n, dr=dr, dt=yee_dt(dr))
    ax = [np.arange(1, m + 1) for m in n]
    mid = [m / 2 + 0.5 for m in n]
    last = n[-1]
    thick = max(2, min(last // 8, 20))
    a0 = last // 2 - thick // 2
    lo, hi = a0, a0 + thick - 1                                     # the medium's extent along the last axis
    mask = np.zeros(n, bool, order="F")
    if c["scene"] == "gold":
        r = min(min(n) // 6, 20)
        lo, hi = int(mid[2]) - r, int(mid[2]) + r
        x, y, z = np.meshgrid(*ax, indexing="ij", sparse=True)
        mask |= (x - mid[0]) ** 2 + (y - mid[1]) ** 2 + (z - mid[2]) ** 2 <= r * r
    elif d == 1:
        mask[lo - 1:hi] = True
    elif c["scene"] == "drude":                                     # a film with a hole every 40 cells
        mask[((ax[0] - 1) % 40) >= 15, lo - 1:hi] = True
    else:                                                           # a pixelated design region, fill 0.4
        box = tuple(slice(m // 4, m // 4 + m // 2) for m in n[:-1]) + (slice(lo - 1, hi),)
        mask[box] = rng.random(mask[box].shape) < 0.4
    s["mask"] = mask
    # the simulation is under way: a smooth field of a few wave lengths in every driven E component
    comps = {1: [EX], 2: [EZ] if c["mode"] == "tmz" else [EX, EY], 3: [EX, EY, EZ]}[d]
    s["fields"] = {}
    for f in comps:
        v = np.array(rng.uniform(0.5, 1.0) * 2e-4)
        for m in n:
            q = np.arange(1, m + 1)
            v = np.multiply.outer(v, np.cos(2 * np.pi * q / rng.uniform(20, 60) + rng.uniform(0, 2 * np.pi)))
        if d == 1:
            v[0] = v[-1] = 0.0
        s["fields"][f] = v
    tau = 5.0 * FS
    comp = {1: 1, 2: 3 if c["mode"] == "tmz" else 1, 3: 1}[d]
    s["src"] = dict(comp=comp, axis=d, index=npml + 4, amp=rng.uniform(0.5, 1.0) * 1e-2, w0=rng.uniform(2.0, 3.0) * EV,
                    t0=0.3 * tau, tau=tau, phase=rng.uniform(0, 2 * np.pi))
    ne = c["emitters"]
    if ne:                                                          # a layer of molecules beside the medium
        zz = min(hi + 4, last - npml - 2)
        if d == 1:
            cells = (zz + np.arange(ne))[:, None]
        elif d == 2:
            cells = np.stack([rng.choice(n[0], ne, replace=ne > n[0]) + 1, np.full(ne, zz)], 1)
        else:
            plane, box = n[0] - 4, (n[0] - 4) * (n[1] - 4)
            p = rng.choice(box * max(2, -(-ne // box)), ne, replace=False)
            cells = np.stack([p % plane + 3, p // plane % (n[1] - 4) + 3, zz + p // box], 1)
        levels = 2 if d < 3 else 3
        u = np.zeros((ne, 3))
        u[:, comp - 1] = 1.0
        t = np.stack([np.full(ne, 1000.0 * FS), np.full(ne, 100.0 * FS)], 1)
        if levels == 2:
            p = np.concatenate([rng.normal(3.0, 0.05, (ne, 1)) * EV, np.full((ne, 1), 10.0 * DEBYE), t, u], 1)
        else:
            p = np.concatenate([rng.normal(2.1, 0.03, (ne, 1)) * EV, rng.normal(2.3, 0.03, (ne, 1)) * EV,
                                rng.uniform(5.0, 8.0, (ne, 2)) * DEBYE, t, u], 1)
        s["emitters"] = dict(cells=cells.astype(np.int32), params=p, levels=levels, density=1e-3 / NM ** 3)
    s["det_field"] = {1: EX, 2: EZ if c["mode"] == "tmz" else HZ, 3: EX}[d]
    s["det"] = np.stack([rng.integers(2, m, 16) for m in n], 1).astype(np.int32)
    s["read"] = {1: [EX, HY], 2: [EZ, HX] if c["mode"] == "tmz" else [EX, HZ], 3: [EX, HY]}[d]
    if np.prod(n) > 4e6:
        s["read"] = s["read"][:1]                                   # one component of the largest grids
    return s


def _sweep_cases(c):
    r = random.Random(c["sides"])
    return [dict(_grid(3, (n, n, n), "full", "fp32", "ccc", c["npml"], c["dr_nm"], "pixels", 0, c["steps"], c["every"]))
            for n in (r.randint(c["lo"], c["hi"]) for _ in range(c["count"]))]


def _solve_inputs(c, seed):
    rng = np.random.default_rng([seed, c["nx"], c["ny"], c["nz"]])
    n = [c["nx"], c["ny"], c["nz"]][:c["dims"]]
    eps = 1.0 + 1.25 * (rng.random(n) < 0.4) + 0.1j
    j = rng.normal(size=[6] + n[::-1])
    return n, eps, j


def _network_inputs(c, seed):
    rng = np.random.default_rng([seed, c["rows"], c["T"]])
    shapes = [(512, 160), (512,), (256, 128), (256,), (256, 256), (256,), (256, 256), (256,), (256,), (1,)]
    p = [rng.uniform(-1, 1, s) / math.sqrt(s[-1]) if len(s) == 2 else np.zeros(s) for s in shapes]
    p[0][256:384, 32:] = 0.0
    p[0][384:, :32] = 0.0
    p[1][128:256] = 1.0
    p[8] = rng.uniform(-1, 1, 256) / 16.0
    # band-limited drives and the response of a damped oscillator to them
    B, L = c["rows"], c["T"] + 31
    t = np.arange(L)
    e = sum(rng.uniform(0.05, 0.2, (B, 1)) * np.cos(rng.uniform(0.05, 0.4, (B, 1)) * t + rng.uniform(0, 6.28, (B, 1)))
            for _ in range(4)).astype(np.float32)
    y, v, x = np.zeros((L, B), np.float32), np.zeros(B), np.zeros(B)
    w = rng.uniform(0.15, 0.25, B)
    for q in range(L):
        v += w * w * (e[:, q] - x) - 0.02 * v
        x = x + v
        y[q] = 0.5 * x
    return [q.astype(np.float32) for q in p], e, np.ascontiguousarray(y[31:])


# ---- the framework's side ----------------------------------------------------------------------
def _medium(scene, dt):
    m = MEDIA[scene]
    if m["kind"] == "dielectric":
        return omx.medium_dielectric(m["eps"])
    if m["kind"] == "drude":
        return omx.medium_drude(m["wp"] * EV, m["gamma"] * EV, m["eps"], dt)
    return omx.medium_dl_custom(m["eps"], m["wp"], m["gamma"], m["poles"], m["strengths"], m["widths"], dt)


def _build(c, s):
    d, n = c["dims"], s["n"]
    g = omx.TMxll(d, n, c["npml"], [KIND[b] for b in c["bnd"]], s["dt"], s["dr"],
                  mode=omx.TEZ if c["mode"] == "tez" else omx.TMZ, precision=c["prec"])
    m = s["mask"].astype(np.int32)
    g.set_media([_medium(c["scene"], s["dt"])], m if d == 1 else np.stack([m, m, m], -1))
    q = s["src"]
    g.add_plane_source(q["comp"], q["axis"], q["index"], q["amp"], q["w0"], q["t0"], q["tau"], 0.0, 1e30, q["phase"])
    e = s.get("emitters")
    group = g.add_q_group(omx.Q_MATERIAL, omx.THREE_LEVEL if e["levels"] == 3 else omx.TWO_LEVEL, e["cells"],
                          e["params"], e["density"], s["dt"]) if e else None
    for p in s["det"]:
        g.add_detector(omx.POINT, s["det_field"], p)
    for f, v in s["fields"].items():
        lo, hi = g.field_bounds(f)
        a = np.zeros([h - b + 1 for b, h in zip(lo, hi)], order="F")
        own = tuple(slice(1 - lo[x], 1 - lo[x] + n[x]) if x < d else slice(0, 1) for x in range(3))
        a[own] = v.reshape(v.shape + (1,) * (3 - d))
        g.write_field(f, a)
    return g, group


def prepare(case, seed):
    c = case
    if c["kind"] == "grid":
        s = _scene(c, seed)
        g, group = _build(c, s)
        return dict(c=c, g=g, group=group, read=s["read"], dt=s["dt"], tt=1)
    if c["kind"] == "sweep":
        members = [(k, _scene(k, seed + 7 * i)) for i, k in enumerate(_sweep_cases(c))]
        grids = [_build(k, s)[0] for k, s in members]
        return dict(c=c, grids=grids, batch=omx.Batch(grids), read=members[0][1]["read"], tt=1)
    if c["kind"] == "solve":
        n, eps, j = _solve_inputs(c, seed)
        op = omx.FDOperator(n, c["npml"], c["nder"], [{"c": 3, "p": 2}[b] for b in c["bnd"]], 0.05, 2 * np.pi / 1.55, eps)
        full = op.zeros()
        full[(slice(None),) + tuple(slice(c["nder"], c["nder"] + m) for m in n[::-1])] = j
        return dict(c=c, op=op, j=full, f0=op.zeros())
    p, e, y = _network_inputs(c, seed)
    return dict(c=c, net=omx.Closure(np.concatenate([q.ravel() for q in p])), e=e, y=y)


def _loop_of_calls(g, group, tt0, steps, every, dt):
    """The reference's time loop in the host program's hands."""
    for tt in range(tt0, tt0 + steps):
        time = dt * (tt - 0.5)
        g.td_propagate_H_field()
        g.source_interactions(time)
        g.td_propagate_E_field(time, time)
        if group is not None:
            g.q_group_step(group, tt)
        if tt % every == 0:
            g.write_detectors_outputs(time)


def _results(g, group, fields, prec):
    # every value of an FP32 grid carries FP32 rounding: they are returned in that type
    real = np.float32 if prec == "fp32" else np.float64
    times, values = g.drain_detectors()
    out = {"times": times, "detectors": values.astype(real), "fields": [g.read_field(f).astype(real, copy=False) for f in fields]}
    if group is not None:
        q = group.read()
        out["dipole"], out["rho"] = q["dipole"].astype(real), q["rho"].astype(real)
    return out


def run(state):
    c = state["c"]
    if c["kind"] == "grid":
        g, tt = state["g"], state["tt"]
        if c["calls"]:
            _loop_of_calls(g, state["group"], tt, c["steps"], c["every"], state["dt"])
        else:
            g.run(tt, c["steps"], 1, c["every"])
        state["tt"] = tt + c["steps"]
        return _results(g, state["group"], state["read"], c["prec"])
    if c["kind"] == "sweep":
        tt = state["tt"]
        state["batch"].run(tt, c["steps"], 1, c["every"])
        state["batch"].synchronize()
        state["tt"] = tt + c["steps"]
        return [_results(g, None, state["read"], "fp32") for g in state["grids"]]
    if c["kind"] == "solve":
        f, _, _, _ = state["op"].solve(state["j"], state["f0"], c["tol"], 2000, c["L"])
        return f
    if c["what"] == "forward":
        return state["net"].forward(state["e"], c["T"])
    loss, grad = state["net"].gradient(state["e"], state["y"], c["skip"])
    return {"loss": np.float32(loss), "grad": grad}


# ---- what a pass cannot do without ---------------------------------------------------------------
def work(case):
    c = case
    if c["kind"] == "grid":
        cells, w = c["nx"] * c["ny"] * c["nz"], 4 if c["prec"] == "fp32" else 8
        comps = {1: 2, 2: 3, 3: 6}[c["dims"]]
        ops = {1: 10, 2: 22, 3: 42}[c["dims"]]
        e = c["emitters"] * c["steps"]
        # each step reads and writes every field value and the emitters' states once
        return {"bytes": 2.0 * w * comps * cells * c["steps"] + e * (200 if c["dims"] == 3 else 120),
                "flops": float(ops * cells * c["steps"] + e * (340 if c["dims"] == 3 else 120))}
    if c["kind"] == "sweep":
        parts = [work(k) for k in _sweep_cases(c)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    if c["kind"] == "solve":
        cells, taps = c["nx"] * c["ny"] * c["nz"], 2 * c["nder"]
        # of the order of 100 outer iterations, each of 2 L operator applications, with the vectors between them
        its = 100.0 * 2 * c["L"]
        return {"bytes": its * cells * 16 * (6 + 6 + 1 + 12), "flops": its * cells * (12 * taps * 4 + 66 + 200)}
    steps = float(c["rows"] * c["T"])
    macs = 512 * 160 + 256 * 128 + 2 * 256 * 256 + 256
    back = 3 if c["what"] == "gradient" else 1
    return {"bytes": 4.0 * (c["rows"] * (c["T"] + 31) + 2 * steps) + 2.0 * macs * back, "flops": 2.0 * macs * steps * back}


# ---- the same results in 64 bits -----------------------------------------------------------------
LEVI = {(0, 1, 2): 1, (1, 2, 0): 1, (2, 0, 1): 1, (0, 2, 1): -1, (2, 1, 0): -1, (1, 0, 2): -1}


def _cpml(npml, dr, dt):
    """Convolutional PML grading (index 1..npml for E, 1..npml-1 for H): b, c, kappa."""
    si = (1 / 1.602176634e-19) ** 2 / 2.4188843265864e-17 / (1 / 9.1093837139e-31 * (1 / 5.29177210544e-11) ** 3)
    smax = float(np.float32(0.8) * np.float32(4.0)) / (dr * math.sqrt(MU0 / EPS0))

    def table(r, ra):
        r3 = float(np.float32(r) ** 3)
        sig, alpha, kap = smax * r3, float(np.float32(0.05)) * si * float(np.float32(ra)), 1 + 4 * r3
        b = math.exp(-(sig / kap + alpha) * dt / EPS0)
        return b, (sig * (b - 1) / (sig + kap * alpha) / kap if sig else 0.0), kap

    e = [table((npml - k) / (npml - 1), (k - 1) / (npml - 1)) for k in range(1, npml + 1)]
    h = [table((npml - k - 0.5) / (npml - 1), (k - 0.5) / (npml - 1)) for k in range(1, npml)]
    return np.array(e), np.array(h)


def _ade(scene, dt):
    """Coefficients of the medium's auxiliary differential equations."""
    m = MEDIA[scene]
    w, gam = m["wp"] * EV, m["gamma"] * EV
    A1, A2 = (2 - gam * dt) / (2 + gam * dt), EPS0 * w * w * dt / (2 + gam * dt)
    al, be, ga = [], [], []
    for p, f, g in zip(m.get("poles", []), m.get("strengths", []), m.get("widths", [])):
        p, g, a = p * EV, g * EV, f * w * w
        al.append((2 - p * p * dt * dt) / (1 + 0.5 * g * dt))
        be.append((g * dt - 2) / (g * dt + 2))
        ga.append(EPS0 * a * dt / (g * dt + 2))
    den = m["eps"] * EPS0 / dt + 0.5 * A2 + 0.5 * sum(ga)
    return dict(A1=A1, A2=A2, C1=(m["eps"] * EPS0 / dt - 0.5 * A2) / den, C2=0.5 * sum(ga) / den, C3=1 / den,
                C4=0.5 * (A1 + 1) / den, al=al, be=be, ga=ga)


class _Yee:
    """The Yee scheme with CPML on padded 64-bit arrays (x, y, z), inactive axes of size one."""

    def __init__(self, c, s):
        self.c, self.s = c, s
        d = c["dims"]
        self.axes = {1: [2], 2: [0, 1], 3: [0, 1, 2]}[d]
        n = [1, 1, 1]
        for a, m in zip(self.axes, s["n"]):
            n[a] = m
        self.n = n
        self.shape = [n[a] + 2 if a in self.axes else 1 for a in range(3)]
        self.E = {b: self.zeros() for b in {"x": [0], "tmz": [2], "tez": [0, 1], "full": [0, 1, 2]}[c["mode"]]}
        self.H = {b: self.zeros() for b in {"x": [1], "tmz": [0, 1], "tez": [2], "full": [0, 1, 2]}[c["mode"]]}
        self.per = [a for a, b in zip(self.axes, c["bnd"]) if b == "p"]
        dt, dr, npml = s["dt"], s["dr"], c["npml"]
        self.dmu, self.deps = dt / MU0, dt / EPS0
        te, th = _cpml(npml, dr, dt)
        self.de, self.dh, self.slabs = {}, {}, {}
        for a, b in zip(self.axes, c["bnd"]):
            m = n[a]
            ke, kh = np.full(m + 1, 1 / dr), np.full(m + 1, 1 / dr)
            if b == "c":
                for k in range(1, npml + 1):
                    ke[k] = 1 / (te[k - 1, 2] * dr)
                    if k < npml:
                        kh[k] = 1 / (th[k - 1, 2] * dr)
                for q, k in enumerate(range(m + 1 - npml, m)):
                    ke[k], kh[k] = 1 / (te[npml - 1 - q, 2] * dr), 1 / (th[npml - 2 - q, 2] * dr)
                self.slabs[a] = {"E": [(2, npml, te[1:npml]), (m + 1 - npml, m - 1, te[1:npml][::-1])],
                                 "H": [(1, npml - 1, th), (m + 1 - npml, m - 1, th[::-1])]}
            self.de[a], self.dh[a] = self.line(ke[1:], a), self.line(kh[1:], a)
        self.psi = {}
        for b, v in s["fields"].items():
            w = torch.as_tensor(v, device="cuda", dtype=torch.float64)
            self.E[b - 1][self.cells()] = w.reshape([n[a] for a in range(3)])
        mask = np.zeros(self.shape, bool)
        mask[self.cells()] = s["mask"].reshape(n)
        mask = torch.as_tensor(mask, device="cuda")
        md = MEDIA[c["scene"]]
        self.eps = torch.where(mask[self.cells()], 1 / md["eps"], 1.0) if md["kind"] == "dielectric" else 1.0
        self.disp = None
        if md["kind"] != "dielectric":
            self.at = mask[self.cells()].reshape(-1).nonzero().reshape(-1)
            self.disp = _ade(c["scene"], dt)
            k = len(self.disp["al"])
            z = lambda: torch.zeros(self.at.numel(), dtype=torch.float64, device="cuda")  # noqa: E731
            self.pol = {b: dict(PD=z(), Eo=z(), P=[z() for _ in range(k)], Po=[z() for _ in range(k)]) for b in self.E}
        self.em = None
        if "emitters" in s:
            self.set_emitters(s["emitters"])

    def zeros(self):
        return torch.zeros(self.shape, dtype=torch.float64, device="cuda")

    def line(self, v, a):
        return torch.as_tensor(np.ascontiguousarray(v), device="cuda", dtype=torch.float64).reshape(
            [-1 if b == a else 1 for b in range(3)])

    def cells(self, a=None, shift=0, lo=None, hi=None):
        """Slices of the cells 1..n of every active axis; along `a` shifted, or lo..hi shifted."""
        out = []
        for b in range(3):
            if b not in self.axes:
                out.append(slice(0, 1))
            elif b == a:
                out.append(slice((lo or 1) + shift, (hi or self.n[b]) + 1 + shift))
            else:
                out.append(slice(1, self.n[b] + 1))
        return tuple(out)

    def plane(self, a, k):
        return tuple(k if b == a else slice(None) for b in range(3))

    def half(self, F, G, den, coef, which, step):
        """rotations of G added to F: step +1 (E differences into H) or -1 (H differences into E)."""
        rot = {}
        for q in F:
            r = None
            for a in self.axes:
                b = 3 - q - a
                if a == q or b not in G:
                    continue
                sign = LEVI[(q, a, b)] * -step
                diff = (G[b][self.cells(a, 1)] - G[b][self.cells()]) if step > 0 else \
                    (G[b][self.cells()] - G[b][self.cells(a, -1)])
                t = sign * diff * den[a]
                r = t if r is None else r + t
            rot[q] = r
        return rot

    def absorb(self, F, G, coef, which, step):
        for q in F:
            for a in self.axes:
                b = 3 - q - a
                if a == q or b not in G or a not in self.slabs:
                    continue
                sign = LEVI[(q, a, b)] * -step
                for i, (lo, hi, t) in enumerate(self.slabs[a][which]):
                    here = self.cells(a, 0, lo, hi)
                    diff = (G[b][self.cells(a, 1, lo, hi)] - G[b][here]) if step > 0 else \
                        (G[b][here] - G[b][self.cells(a, -1, lo, hi)])
                    key = (which, q, a, i)
                    bb, cc = self.line(t[:, 0], a), self.line(t[:, 1], a)
                    if key not in self.psi:
                        self.psi[key] = torch.zeros_like(diff)
                    self.psi[key] = bb * self.psi[key] + cc * (sign * diff) / self.s["dr"]
                    F[q][here] += coef * self.psi[key]

    def wrap(self, F, lo):
        for a in self.per:
            for v in F.values():
                if lo:
                    v[self.plane(a, 0)] = v[self.plane(a, self.n[a])]
                else:
                    v[self.plane(a, self.n[a] + 1)] = v[self.plane(a, 1)]

    def step(self, tt):
        c, s, d1 = self.c, self.s, self.c["dims"] == 1
        time = s["dt"] * (tt - 0.5)
        self.wrap(self.E, False)
        for q, r in self.half(self.H, self.E, self.dh, self.dmu, "H", 1).items():
            if d1:
                r[:, :, -1] = 0.0
            self.H[q][self.cells()] += self.dmu * r
        self.absorb(self.H, self.E, self.dmu, "H", 1)
        q = s["src"]
        amp = q["amp"] * math.exp(-((time - q["t0"]) / q["tau"]) ** 2) * math.cos(q["w0"] * (time - q["t0"]) + q["phase"])
        ax = self.axes[-1]
        self.E[q["comp"] - 1][self.cells(ax, 0, q["index"], q["index"])] += self.deps / s["dr"] / C0 / 2 * amp
        self.wrap(self.H, True)
        for b, r in self.half(self.E, self.H, self.de, self.deps, "E", -1).items():
            here = self.E[b][self.cells()]
            old = here.reshape(-1)[self.at] if self.disp else None
            if d1:
                r[:, :, 0] = 0.0
                r[:, :, -1] = 0.0
            new = here + self.deps * self.eps * r
            if self.em is not None and b == self.em["comp"]:
                J = self.em["Jo"]                    # the step time equals the emitters' last time stamp
                if len(self.axes) == 1 or c["mode"] == "tmz":
                    new -= self.deps * J[self.cells()]
                else:
                    new -= self.deps * 0.5 * (J[self.cells()] + J[self.cells(b, 1)])
            if self.disp:
                new.reshape(-1)[self.at] = self.polarise(b, old, r.reshape(-1)[self.at])
            self.E[b][self.cells()] = new
        self.absorb(self.E, self.H, self.deps, "E", -1)
        if self.em is not None:
            self.emit()

    def polarise(self, b, E, rot):
        k, p = self.disp, self.pol[b]
        new = k["C1"] * E + k["C2"] * p["Eo"] + k["C3"] * rot - k["C4"] * p["PD"]
        for al, be, P, Po in zip(k["al"], k["be"], p["P"], p["Po"]):
            new = new - 0.5 * (1 + al) * k["C3"] * P - 0.5 * be * k["C3"] * Po
        p["PD"] = k["A1"] * p["PD"] + k["A2"] * (new + E)
        nxt = [al * P + be * Po + ga * (new - p["Eo"]) for al, be, ga, P, Po in
               zip(k["al"], k["be"], k["ga"], p["P"], p["Po"])]
        p["Eo"], p["Po"], p["P"] = E, p["P"], nxt
        return new

    def set_emitters(self, e):
        t = lambda v: torch.as_tensor(v, device="cuda", dtype=torch.float64)  # noqa: E731
        pad = [np.ones(len(e["cells"]), np.int64) * 0] * 3
        for x, a in enumerate(self.axes):
            pad[a] = e["cells"][:, x].astype(np.int64)
        flat = (pad[0] * self.shape[1] + pad[1]) * self.shape[2] + pad[2]
        _, first = np.unique(flat[::-1], return_index=True)          # the last writer of a cell wins
        keep = np.sort(len(flat) - 1 - first)
        comp = int(np.argmax(e["params"][0, -3:]))
        self.em = dict(comp=comp, flat=torch.as_tensor(flat, device="cuda"), keep=torch.as_tensor(keep, device="cuda"),
                       p=t(e["params"]).T, levels=e["levels"], rho=t(np.zeros((3 if e["levels"] == 2 else 8, len(flat)))),
                       J=self.zeros(), Jo=self.zeros(), dip=t(np.zeros(len(flat))), density=e["density"])

    def emit(self):
        m, dt = self.em, self.s["dt"]
        E = self.E[m["comp"]].reshape(-1)
        stride = [self.shape[1] * self.shape[2], self.shape[2], 1][m["comp"]]
        F = E[m["flat"]] if len(self.axes) == 1 or self.c["mode"] == "tmz" else 0.5 * (E[m["flat"] - stride] + E[m["flat"]])
        p, f = m["p"], (self.rhs2 if m["levels"] == 2 else self.rhs3)
        r = m["rho"]
        k1 = f(p, F, r)
        k2 = f(p, F, r + 0.5 * dt * k1)
        k3 = f(p, F, r + 0.5 * dt * k2)
        k4 = f(p, F, r + dt * k3)
        m["rho"] = r = r + dt / 6 * (k1 + 2 * k2 + 2 * k3 + k4)
        dip = 2 * p[1] * r[1] if m["levels"] == 2 else 2 * p[2] * r[2] + 2 * p[3] * r[4]
        m["Jo"].copy_(m["J"])
        m["J"].reshape(-1)[m["flat"][m["keep"]]] = (m["density"] * (dip - m["dip"]) / dt)[m["keep"]]
        m["dip"] = dip

    @staticmethod
    def rhs2(p, E, r):
        g = p[1] * E
        return torch.stack([2 * g * r[2] - r[0] / p[2], p[0] * r[2] - r[1] / p[3],
                            -p[0] * r[1] + g * (1 - 2 * r[0]) - r[2] / p[3]])

    @staticmethod
    def rhs3(p, E, r):
        e1, e2, g1, g2, i1, i2 = p[0], p[1], p[2] * E, p[3] * E, 1 / p[4], 1 / p[5]
        p0 = 1 - r[0] - r[1]
        return torch.stack([
            2 * g1 * r[3] - r[0] * i1, 2 * g2 * r[5] - r[1] * i1,
            e1 * r[3] - g2 * r[7] - r[2] * i2, -e1 * r[2] + g1 * (p0 - r[0]) - g2 * r[6] - r[3] * i2,
            e2 * r[5] + g1 * r[7] - r[4] * i2, -e2 * r[4] + g2 * (p0 - r[1]) - g1 * r[6] - r[5] * i2,
            (e2 - e1) * r[7] + g2 * r[3] + g1 * r[5] - r[6] * i2, -(e2 - e1) * r[6] + g2 * r[2] - g1 * r[4] - r[7] * i2])

    def sample(self):
        d, f = self.c["dims"], self.s["det_field"]
        ix = [np.zeros(len(self.s["det"]), np.int64)] * 3
        for x, a in enumerate(self.axes):
            ix[a] = self.s["det"][:, x].astype(np.int64)
        ix = [torch.as_tensor(v, device="cuda") for v in ix]
        if f == HZ:
            h = self.H[2]
            return 0.25 * (h[ix[0], ix[1], ix[2]] + h[ix[0] - 1, ix[1], ix[2]] + h[ix[0], ix[1] - 1, ix[2]] +
                           h[ix[0] - 1, ix[1] - 1, ix[2]])
        v = self.E[f - 1]
        if d == 3:
            return 0.5 * (v[ix[0] - 1, ix[1], ix[2]] + v[ix[0], ix[1], ix[2]])
        return v[ix[0], ix[1], ix[2]]

    def snapshot(self, f):
        """A field over the reference's bounds: E ghosts are zero, H ghosts 0 of periodic axes wrap."""
        n, d1 = self.n, self.c["dims"] == 1
        q = (f - 1) % 3
        if f <= 3:
            v = torch.zeros_like(self.E[q])
            v[self.cells()] = self.E[q][self.cells()]
        else:
            v = self.H[q]
        out = []
        for a in range(3):
            if a not in self.axes:
                out.append(slice(0, 1))
            elif d1:
                out.append(slice(1, n[a] + 1) if f <= 3 else slice(1, n[a]))
            elif f <= 3:
                out.append(slice(0, n[a] + 1) if a == q else slice(1, n[a] + 2))
            else:
                out.append(slice(1, n[a] + 1) if a == q else slice(0, n[a] + 1))
        v = v[tuple(out)]
        return v.reshape(-1, 1, 1) if d1 else v

    def results(self):
        c, s = self.c, self.s
        times, values = [], []
        for tt in range(1, c["steps"] + 1):
            self.step(tt)
            if tt % c["every"] == 0:
                times.append(s["dt"] * (tt - 0.5))
                values.append(self.sample())
        host = lambda v: v.cpu().numpy()  # noqa: E731
        out = {"times": np.array(times), "detectors": host(torch.stack(values)),
               "fields": [host(self.snapshot(f)) for f in s["read"]]}
        if self.em is not None:
            dip = np.zeros((len(self.em["dip"]), 3))
            dip[:, self.em["comp"]] = host(self.em["dip"])
            out["dipole"], out["rho"] = dip, host(self.em["rho"].T)
        return out


def _solution(c, seed):
    """The solution of the frequency-domain system by GMRES to 1e-11 of the right-hand side."""
    n, eps, j = _solve_inputs(c, seed)
    w0, dr, g, d = 2 * np.pi / 1.55, 0.05, c["nder"], c["dims"]
    cx = lambda v: torch.as_tensor(v, device="cuda", dtype=torch.complex128)  # noqa: E731
    coef = {1: [0.5], 2: [2 / 3, -1 / 12], 3: [3 / 4, -3 / 20, 1 / 60]}[g]
    sinv = []
    for a in range(d):
        v = np.ones(n[a], complex)
        if c["bnd"][a] == "c":
            for i in range(1, c["npml"] + 1):
                r = ((c["npml"] - i + 1) / c["npml"]) ** 3
                v[i - 1] = v[n[a] - i] = 1 / ((1 + 4 * r) - 1j * 3.2 / dr * r / w0)
        sinv.append(cx(v).reshape([-1 if d - 1 - a == q else 1 for q in range(d)]))
    med = cx(-0.5j * w0 * (eps.transpose() - 1.0))
    shape = j.shape
    axis_of = lambda a: d - 1 - a  # noqa: E731  (arrays are z, y, x)

    def der(v, a, q):
        ax, m = axis_of(a), n[a]
        lo, hi = torch.zeros_like(v.narrow(ax, 0, g)), torch.zeros_like(v.narrow(ax, 0, g))
        if c["bnd"][a] == "p":
            if d == 2 or a != 1 or q != 4:
                lo = v.narrow(ax, m - g, g)
            if d == 2 or a != 1 or q != 3:
                hi = v.narrow(ax, 0, g)
        w = torch.cat([lo, v, hi], ax)
        return sum(k / dr * (w.narrow(ax, g + t, m) - w.narrow(ax, g - t, m)) for t, k in enumerate(coef, 1)) * sinv[a]

    def apply(x):
        f = x.reshape(shape)
        e = [med * (f[q] + f[q + 3]) for q in range(3)]
        out = []
        for h in range(2):
            s = 1j if h == 0 else -1j
            s = s if d == 3 else -s
            for q in range(3):
                t = 0
                for a in range(d):
                    b = 3 - q - a
                    if a != q and 0 <= b < 3:
                        t = t + LEVI[(q, a, b)] * der(f[b + 3 * h], a, b + 3 * h)
                out.append(s * t - 1j * w0 * f[q + 3 * h] + e[q])
        return torch.stack(out).reshape(-1)

    rhs = cx(j).reshape(-1)
    beta = float(torch.linalg.norm(rhs))
    most = 2500
    V = torch.empty((most + 1, rhs.numel()), dtype=torch.complex128, device="cuda")
    R = np.zeros((most + 1, most), complex)
    cs, sn, q = np.zeros(most), np.zeros(most, complex), np.zeros(most + 1, complex)
    V[0], q[0] = rhs / beta, beta
    k = 0
    while k < most and abs(q[k]) > 1e-11 * beta:
        w = apply(V[k])
        h = torch.zeros(k + 1, dtype=torch.complex128, device="cuda")
        for _ in range(2):
            t = V[:k + 1].conj() @ w
            w = w - t @ V[:k + 1]
            h += t
        col = h.cpu().numpy()
        nw = float(torch.linalg.norm(w))
        V[k + 1] = w / nw
        for i in range(k):
            col[i], col[i + 1] = cs[i] * col[i] + sn[i] * col[i + 1], -np.conj(sn[i]) * col[i] + cs[i] * col[i + 1]
        r = math.hypot(abs(col[k]), nw)
        ph = col[k] / abs(col[k])
        cs[k], sn[k] = abs(col[k]) / r, ph * nw / r
        col[k] = ph * r
        R[:k + 1, k] = col
        q[k], q[k + 1] = cs[k] * q[k], -np.conj(sn[k]) * q[k]
        k += 1
    y = np.linalg.solve(R[:k, :k], q[:k])
    x = (cx(y) @ V[:k]).reshape(shape).cpu().numpy()
    pad = [s + (2 * g if i else 0) for i, s in enumerate(shape)]
    out = np.zeros(pad, complex)
    out[(slice(None),) + tuple(slice(g, g + m) for m in n[::-1])] = x
    return out


def _network(c, seed):
    p, e, y = _network_inputs(c, seed)
    t64 = lambda v: torch.as_tensor(v, device="cuda", dtype=torch.float64)  # noqa: E731
    p, e, y = [t64(v).requires_grad_(c["what"] == "gradient") for v in p], t64(e), t64(y)
    Wg, bg, W1, b1, W2, b2, W3, b3, w4, b4 = p
    keep = torch.ones_like(Wg)
    keep[256:384, 32:] = 0
    keep[384:, :32] = 0
    h, out = torch.zeros((c["rows"], 128), dtype=torch.float64, device="cuda"), []
    for t in range(c["T"]):
        G = torch.cat([e[:, t:t + 32], h], 1) @ (Wg * keep).T + bg
        r, z = torch.sigmoid(G[:, :128]), torch.sigmoid(G[:, 128:256])
        h = (1 - z) * torch.tanh(G[:, 256:384] + r * G[:, 384:]) + z * h
        a = torch.tanh(torch.tanh(torch.tanh(h @ W1.T + b1) @ W2.T + b2) @ W3.T + b3)
        out.append(a @ w4 + b4)
    out = torch.stack(out)
    if c["what"] == "forward":
        return out.cpu().numpy()
    loss = ((out - y)[c["skip"]:] ** 2).mean()
    grad = torch.autograd.grad(loss, p)
    return {"loss": np.float64(loss.item()), "grad": torch.cat([v.reshape(-1) for v in grad]).cpu().numpy()}


def exact(case, seed):
    c = case
    if c["kind"] == "grid":
        return _Yee(c, _scene(c, seed)).results()
    if c["kind"] == "sweep":
        return [_Yee(k, _scene(k, seed + 7 * i)).results() for i, k in enumerate(_sweep_cases(c))]
    if c["kind"] == "solve":
        return _solution(c, seed)
    return _network(c, seed)
