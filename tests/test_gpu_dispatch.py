"""Kernel variants chosen by size, type and alignment, at the sizes where a choice or its remainder
can go wrong, against the FP64 oracle or the general path."""
import numpy as np
import pytest

import omx

pytestmark = pytest.mark.gpu


def seeded_pair(orc, dims, n, npml, bnd, dr, mode, amp, seed, precision="fp64"):
    """A library grid and an oracle grid with the same random E fields of amplitude amp."""
    dt = omx.units.yee_dt(dr)
    gpu = omx.TMxll(dims, n, npml, bnd, dt, dr, mode=mode, precision=precision)
    cpu = orc.Grid(dims, n, npml, bnd, dt, dr, mode=mode)
    rng = np.random.default_rng(seed)
    comps = {1: [1], 2: [3] if mode == omx.TMZ else [1, 2], 3: [1, 2, 3]}[dims]
    for f in comps:
        lo, hi = gpu.field_bounds(f)
        a = np.zeros([h - b + 1 for b, h in zip(lo, hi)], order="F")
        own = tuple(slice(1 - lo[x], 1 - lo[x] + n[x]) if x < dims else slice(None) for x in range(3))
        a[own] = amp * rng.standard_normal(a[own].shape) * (rng.random(a[own].shape) < 0.8)
        if dims == 1:
            a[0] = a[-1] = 0.0
        gpu.write_field(f, a)
        cpu.write_field(f, a)
    return gpu, cpu, dt


def advance(gpu, cpu, dt, steps, calls=False):
    if calls:
        for tt in range(1, steps + 1):
            gpu.td_propagate_H_field()
            gpu.source_interactions(dt * (tt - 0.5))
            gpu.td_propagate_E_field(dt * (tt - 0.5), 0.0)
    else:
        gpu.run(1, steps)
    for tt in range(1, steps + 1):
        cpu.td_propagate_H_field()
        cpu.td_propagate_E_field(dt * (tt - 0.5), 0.0)


FIELDS_OF = {(1, 1): [1, 5], (2, 1): [3, 4, 5], (2, 2): [1, 2, 6], (3, 1): [1, 2, 3, 4, 5, 6]}


# sizes at the edges of the blocks (8 x 16 cells), of the marches (1..16 planes, 1..8 rows)
# and of the CPML slabs
@pytest.mark.parametrize("dims,n,npml,bnd,mode", [
    (1, (64,), 6, (3, 1, 1), 1),
    (2, (129, 33), 5, (3, 3, 1), 1),
    (2, (17, 9), 3, (2, 3, 1), 2),
    (2, (127, 70), 5, (2, 3, 1), 2),
    (2, (640, 641), 6, (3, 2, 1), 2),
    (2, (8, 70001), 3, (2, 3, 1), 1),        # more rows than a launch takes blocks along y
    (3, (33, 29, 26), 4, (3, 3, 3), 1),
    (3, (7, 16, 9), 3, (2, 3, 1), 1),
    (3, (31, 17, 65), 5, (2, 3, 3), 1),
])
# amplitudes where quotients by dr are ordinary, and down to where they or their remainders leave
# the normal range; spacings with short and with full mantissas
@pytest.mark.parametrize("amp,dr", [(1.0, 37.794522518155646), (1e-250, 19.0), (3e-306, 0.7), (1e280, 1.0 / 3.0)])
def test_fp64_passes_bit_identical(orc, dims, n, npml, bnd, mode, amp, dr):
    gpu, cpu, dt = seeded_pair(orc, dims, n, npml, bnd, dr, mode, amp, sum(n))
    advance(gpu, cpu, dt, 5)
    for f in FIELDS_OF[(dims, mode)]:
        a, b = gpu.read_field(f), cpu.read_field(f)
        lo, _ = gpu.field_bounds(f)
        own = tuple(slice(1 - lo[x], 1 - lo[x] + n[x]) if x < dims else slice(None) for x in range(3))
        assert np.array_equal(a[own], b[own])
        assert amp < 1e-300 or np.max(np.abs(b[own])) > 0
    gpu.kill()


def test_more_planes_than_blocks_along_z(orc):
    """A grid with more planes (3D) or FP32 rows (2D) than a launch takes blocks along z or y."""
    gpu, cpu, dt = seeded_pair(orc, 3, (4, 3, 66001), 2, (1, 1, 1), 19.0, omx.TMZ, 1.0, 3)
    advance(gpu, cpu, dt, 2)
    assert np.array_equal(gpu.read_field(1), cpu.read_field(1))
    gpu, cpu, dt = seeded_pair(orc, 2, (9, 66003), 3, (1, 3, 1), 19.0, omx.TEZ, 1.0, 4, "fp32")
    advance(gpu, cpu, dt, 2)
    assert np.max(np.abs(gpu.read_field(6) - cpu.read_field(6))) < 1e-5 * np.max(np.abs(cpu.read_field(6)))


@pytest.mark.parametrize("dims,n,bnd,mode,field,precision", [
    (1, (2_200_003,), (3, 1, 1), 1, 1, "fp64"),           # one row longer than a chunk of the staging buffer
    (2, (1701, 1301), (2, 3, 1), 1, 3, "fp32"),           # two chunks, the second partial; periodic ghost column
    (2, (5, 3), (1, 1, 1), 2, 6, "fp64"),
    (3, (131, 129, 130), (2, 2, 2), 1, 2, "fp32"),
    (3, (131, 129, 130), (3, 3, 3), 1, 5, "fp64"),
])
def test_field_round_trip(dims, n, bnd, mode, field, precision):
    """omx_write_field then omx_read_field returns the values, the E ghosts of periodic axes as zero."""
    g = omx.TMxll(dims, n, 4, bnd, 0.07, 19.0, mode=mode, precision=precision)
    lo, hi = g.field_bounds(field)
    shape = [h - b + 1 for b, h in zip(lo, hi)]
    a = np.asfortranarray(np.random.default_rng(1).standard_normal(shape).astype(np.float32).astype(np.float64))
    g.write_field(field, a)
    want = a.copy(order="F")
    for x in range(dims):
        if field <= 3 and bnd[x] == 2 and hi[x] == n[x] + 1:
            want[tuple(-1 if y == x else slice(None) for y in range(3))] = 0.0
    assert np.array_equal(g.read_field(field), want)
    g.kill()


@pytest.mark.parametrize("model,n", [(1, 1), (1, 9), (1, 8192), (1, 8193), (2, 1), (2, 5), (2, 6144), (2, 6145)])
def test_emitter_forms_bit_identical(orc, model, n):
    """One lane per state word up to a number of emitters, one thread per emitter above: the first
    and last sizes of each, partly filled warps."""
    gpu, cpu, dt = seeded_pair(orc, 3, (20, 18, 22), 3, (3, 2, 1), 37.8, omx.TMZ, 1e-3, n)
    rng = np.random.default_rng(n)
    cells = np.stack([rng.integers(2, m, n) for m in (20, 18, 22)], 1).astype(np.int32)
    u = rng.standard_normal((n, 3))
    levels = [rng.uniform(0.05, 0.12, n) for _ in range(model)]
    mu = [rng.uniform(1.0, 4.0, n) for _ in range(model)]
    par = np.stack(levels + mu + [rng.uniform(2e3, 4e4, n), rng.uniform(1e3, 4e3, n)], 1)
    par = np.concatenate([par, u / np.linalg.norm(u, axis=1, keepdims=True)], 1)
    gg = gpu.add_q_group(omx.Q_MATERIAL, model, cells, par, 1e-6, dt)
    before = gg.read()
    for tt in range(1, 4):
        gpu.run(tt, 1)
        a = gg.read()
        E_u = par[:, -3] * a["E"][:, 0] + par[:, -2] * a["E"][:, 1] + par[:, -1] * a["E"][:, 2]
        rho = np.array([orc.emitter_step(model, par[e], before["rho"][e], E_u[e], dt) for e in range(n)])
        d = 2.0 * par[:, 1] * rho[:, 1] if model == 1 else 2.0 * par[:, 2] * rho[:, 2] + 2.0 * par[:, 3] * rho[:, 4]
        dip = d[:, None] * par[:, -3:]
        assert np.array_equal(a["rho"], rho) and np.max(np.abs(rho)) > 0
        assert np.array_equal(a["dipole"], dip)
        assert np.array_equal(a["dPt_dt"], (dip - before["dipole"]) / dt)
        before = a
    gpu.kill()


def bicgstab_rows(O, own, j, f0, L, its):
    """BiCGStab(L) (bicgstab_mod.f90:76-243) with the oracle's operator, FP64 operations written out,
    and the dot products in the library's order: per row of cells, 128 interleaved sums (components
    outermost) halved together, then the rows one after the other.  Returns (f, |r| / |j|)."""
    def mul(a, v):                                           # complex a times a vector (re, im)
        return a[0] * v[0] - a[1] * v[1], a[0] * v[1] + a[1] * v[0]

    def cmul(a, b):
        return a[0] * b[0] - a[1] * b[1], a[0] * b[1] + a[1] * b[0]

    def cdiv(a, b):
        if abs(b[0]) < abs(b[1]):
            t = b[0] / b[1]
            d = b[0] * t + b[1]
            return (a[0] * t + a[1]) / d, (a[1] * t - a[0]) / d
        t = b[1] / b[0]
        d = b[1] * t + b[0]
        return (a[1] * t + a[0]) / d, (a[1] - a[0] * t) / d

    def neg(a):
        return a[0] * -1.0, a[1] * -1.0

    def axpy(v, w, a):                                       # v + a w
        m = mul(a, w)
        return v[0] + m[0], v[1] + m[1]

    def dot(a, b):
        re = a[0] * b[0] - (-a[1]) * b[1]
        im = a[0] * b[1] + (-a[1]) * b[0]
        tot = []
        for p in (re, im):
            nx = p.shape[-1]
            q = np.zeros((p.shape[0], p[0].size // nx, -(-nx // 128) * 128))
            q[:, :, :nx] = p.reshape(p.shape[0], -1, nx)
            s = np.zeros((q.shape[1], 128))
            for c in range(q.shape[0]):
                for x in range(0, q.shape[2], 128):
                    s = s + q[c, :, x:x + 128]
            o = 64
            while o:
                s = s[:, :o] + s[:, o:2 * o]
                o //= 2
            t = 0.0
            for v in s[:, 0]:
                t = t + float(v)
            tot.append(t)
        return tuple(tot)

    def A(v):
        x = np.zeros(j.shape, complex)
        x[own].real, x[own].imag = v
        y = O.apply(x)[own]
        return y.real.copy(), y.imag.copy()

    split = lambda v: (v[own].real.copy(), v[own].imag.copy())  # noqa: E731
    jv, x = split(j), split(f0)
    r0 = axpy(jv, A(x), (-1.0, 0.0))
    zero = (np.zeros_like(jv[0]), np.zeros_like(jv[0]))
    r, u = [r0] + [zero] * L, [zero] * (L + 1)
    r0 = mul((1.0 / np.sqrt(dot(r0, r0)[0]), 0.0), r0)
    nj = np.sqrt(dot(jv, jv)[0])
    rho0, alpha, omega = (1.0, 0.0), (1.0, 0.0), (1.0, 0.0)
    for _ in range(its):
        rho0 = cmul(neg(omega), rho0)
        for q in range(L):
            rho1 = dot(r0, r[q])
            beta = neg(cdiv(cmul(alpha, rho1), rho0))
            rho0 = rho1
            for i in range(q + 1):
                m = mul(beta, u[i])
                u[i] = (m[0] + r[i][0], m[1] + r[i][1])
            u[q + 1] = A(u[q])
            alpha = cdiv(rho0, dot(r0, u[q + 1]))
            for i in range(q + 1):
                r[i] = axpy(r[i], u[i + 1], neg(alpha))
            r[q + 1] = A(r[q])
            x = axpy(x, u[0], alpha)
        tau, sig, gp = {}, [None] * (L + 1), [None] * (L + 1)
        for q in range(1, L + 1):
            for i in range(1, q):
                tau[i, q] = cdiv(dot(r[i], r[q]), sig[i])
                r[q] = axpy(r[q], r[i], neg(tau[i, q]))
            sig[q] = dot(r[q], r[q])
            gp[q] = cdiv(dot(r[q], r[0]), sig[q])
        gam = gp[:]
        omega = gam[L]
        for q in range(L - 1, 0, -1):
            for i in range(q + 1, L + 1):
                m = cmul(tau[q, i], gam[i])
                gam[q] = (gam[q][0] - m[0], gam[q][1] - m[1])
        gpp = [None] * (L + 1)
        for q in range(1, L):
            gpp[q] = gam[q + 1]
            for i in range(q + 1, L):
                m = cmul(tau[q, i], gam[i + 1])
                gpp[q] = (gpp[q][0] + m[0], gpp[q][1] + m[1])
        x = axpy(x, r[0], gam[1])
        r[0] = axpy(r[0], r[L], neg(gp[L]))
        u[0] = axpy(u[0], u[L], neg(gam[L]))
        for q in range(1, L):
            u[0] = axpy(u[0], u[q], neg(gam[q]))
            x = axpy(x, r[q], gpp[q])
            r[0] = axpy(r[0], r[q], neg(gp[q]))
        err = np.sqrt(dot(r[0], r[0])[0])
    return x[0] + 1j * x[1], err / nj


# row lengths at the edges of the thread groups per row (32, 64, 128) and of the split of long rows
# (256); every stencil order; PML, periodic and closed faces
@pytest.mark.parametrize("n,n_der,bnd", [
    ((32, 5, 4), 1, (2, 2, 2)), ((33, 6, 7), 2, (3, 2, 1)), ((64, 4, 5), 3, (1, 2, 2)), ((65, 8, 8), 4, (2, 2, 2)),
    ((128, 9), 2, (3, 2)), ((129, 7), 1, (2, 2)), ((256, 6), 3, (2, 3)), ((257, 5), 2, (2, 2)), ((300, 9), 4, (3, 2)),
    ((31,), 2, (2,)), ((257,), 4, (3,)),
])
def test_fd_rows(orc, n, n_der, bnd):
    """The solver's fused passes against the oracle: the operator bit for bit, infinities and NaN
    included; two iterations of the solver bit for bit against the same recursion."""
    rng = np.random.default_rng(sum(n) + n_der)
    eps = 1.0 + 1.25 * (rng.random(n) < 0.4) + 0.3j
    G = omx.FDOperator(n, 2, n_der, bnd, 0.25, 1.3, eps)
    O = orc.FDOperator(n, 2, n_der, bnd, 0.25, 1.3, eps)
    own = (slice(None),) + tuple(slice(n_der, n_der + m) for m in reversed(n))
    f = G.zeros()
    f[own] = rng.normal(size=f[own].shape) + 1j * rng.normal(size=f[own].shape)
    for transpose in (False, True):
        assert np.array_equal(G.apply(f, transpose)[own], O.apply(f, transpose)[own])
    bad = f.copy()
    flat = bad[own].reshape(-1).copy()
    for q, v in zip(rng.choice(flat.size, 4, replace=False), (np.inf, -np.inf, np.nan, 1e308)):
        flat[q] = v + 1j * flat[q].imag
    bad[own] = flat.reshape(bad[own].shape)
    with np.errstate(all="ignore"):
        assert np.array_equal(G.apply(bad)[own], O.apply(bad)[own], equal_nan=True)
    j = G.zeros()
    j[own] = rng.normal(size=j[own].shape)
    for L in (1, 2, 3):
        got, _, err, its = G.solve(j, f, 1e-30, 1, L)        # two outer iterations
        want, werr = bicgstab_rows(O, own, j, f, L, 2)
        assert its == 2 and err == werr
        assert np.array_equal(got[own], want)
    G.kill()


# tiles cut by every edge (32 x 4 columns in place, 32 x 8 staged), periodic z, single and several
# sources, detectors of E only and of H
@pytest.mark.parametrize("n,bnd,src,taps_h", [
    ((40, 36, 28), (3, 3, 3), "plane", False), ((33, 29, 31), (3, 3, 3), "radial", True),
    ((65, 30, 26), (3, 3, 2), "plane", True), ((31, 37, 40), (1, 3, 1), "both", False),
])
def test_inplace_and_staged_3d_steps_bit_identical(n, bnd, src, taps_h):
    """The FP32 3D step in place (two plain passes) and staged, through graphs, single launches,
    one-step calls and the per-call sequence: every field, record and emitter bit for bit."""
    from test_gpu_parity import fused3_deck
    from gpu_harness import step_loop
    from omx import decks

    deck = fused3_deck(n, bnd, src=src)
    steps = 23
    out = []
    for shape, mode in ((8064, "graph"), (None, "graph"), (None, "plain"), (None, "one"), (None, "calls"),
                        (1, "graph"), (4, "one"), (16, "graph")):
        g = omx.TMxll(3, deck["grid_Ndims"], deck["npml"], deck["boundaries"], deck["dt"], deck["dr"],
                      precision="fp32")
        groups = decks.apply_deck(g, deck, omx, decks.media_map(deck, omx.media_map_from_voxels))
        for det in deck["detectors"]:
            g.add_detector(det["type"], det["field"], det["idx"])
        if taps_h:
            g.add_detector(omx.POINT, "Hy", np.array([[n[0] // 2, n[1] // 2, 12]]))
        if shape:
            g.set_launch_shape(shape)
        if mode == "calls":
            step_loop(g, deck, groups, 1, steps, {"tq_old": 0, "t_skip": 0.0},
                      sample=lambda t: g.write_detectors_outputs(t))
        elif mode == "one":
            for tt in range(1, steps + 1):
                g.run(tt, 1, deck["n_skip"], 1)
        else:
            g.run(1, steps, deck["n_skip"], 1, use_graph=mode == "graph")
        out.append([g.drain_detectors()[1]] + [g.read_field(f) for f in range(1, 7)] +
                   [q for gr in groups for q in (gr.read()["rho"], gr.read()["dipole"])])
        g.kill()
    assert np.max(np.abs(out[0][0])) > 0
    for o in out[1:]:
        assert len(o) == len(out[0])
        for a, b in zip(o, out[0]):
            assert np.array_equal(a, b)


def test_inplace_batch_equals_solo_and_staged():
    """A batch of small grids steps in place in one launch per half step: ragged sides, dispersive
    cells, a folded plane source and radial ones, emitters; equal to solo runs and to the staged
    batch bit for bit, also when the batch is autotuned or switched between calls."""
    from test_gpu_parity import fused3_deck
    from omx import decks

    specs = [((33, 30, 27), (3, 3, 3), "plane"), ((40, 36, 28), (3, 3, 2), "both"), ((29, 41, 26), (1, 3, 3), "plane")]

    def build(spec):
        d = fused3_deck(*spec[:2], src=spec[2])
        g = omx.TMxll(3, d["grid_Ndims"], d["npml"], d["boundaries"], d["dt"], d["dr"], precision="fp32")
        gr = decks.apply_deck(g, d, omx, decks.media_map(d, omx.media_map_from_voxels))
        for det in d["detectors"]:
            g.add_detector(det["type"], det["field"], det["idx"])
        return g, gr

    def state(g, gr):
        return [g.drain_detectors()[1]] + [g.read_field(f) for f in range(1, 7)] + [q.read()["rho"] for q in gr]

    want = []
    for sp in specs:
        g, gr = build(sp)
        g.run(1, 31, 1, 1)
        want.append(state(g, gr))
        g.kill()
    for mode in ("inplace", "staged", "tuned", "switched"):
        grids = [build(sp) for sp in specs]
        b = omx.Batch([g for g, _ in grids])
        if mode == "tuned":
            b.autotune(reps=1)
        if mode == "staged":
            b.set_launch_shape(8016)
        b.run(1, 14, 1, 1)
        if mode == "switched":
            b.synchronize()
            b.set_launch_shape(8016)
        b.run(15, 17, 1, 1)
        b.synchronize()
        for (g, gr), w in zip(grids, want):
            got = state(g, gr)
            assert np.max(np.abs(w[0])) > 0
            for x, y in zip(got, w):
                assert np.array_equal(x, y)
        b.kill()
        for g, _ in grids:
            g.kill()


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
@pytest.mark.parametrize("n,bnd,skip", [
    (64, 3, 1), (71, 1, 2),
    (3072, 3, 1),                            # eight blocks of 384 cell threads: one cell each
    (3073, 3, 2), (3079, 1, 1), (6151, 3, 1),
])
def test_one_launch_1d_loop(n, bnd, skip, precision):
    """The 1D time loop in one launch against one launch per phase, bit for bit: a dielectric, a
    Drude and a Drude-Lorentz layer, two groups that share cells (one inside a layer), three sources
    on one cell or side by side, samples, several calls."""
    ev, fs = omx.UNITS["ev_to_au"], omx.UNITS["fs_to_au"]
    dr = 18.9
    dt = omx.units.yee_dt(dr)
    q = n // 8
    m = np.zeros(n, np.int32)
    m[4 * q:4 * q + 5], m[5 * q:5 * q + 4], m[6 * q:6 * q + 3] = 1, 2, 3
    out = []
    for graph in (True, False):
        g = omx.TMxll(1, (n,), 5, (bnd, 1, 1), dt, dr, precision=precision)
        g.set_media([omx.medium_dielectric(4.0), omx.medium_drude(9.17 * ev, 0.02 * ev, 1.0, dt),
                     omx.medium_dl_custom(5.9, 9.0, 0.07, [2.7, 3.9], [1.0, 0.6], [0.3, 0.5], dt)], m)
        g.add_plane_source(1, 1, 3 * q, 1e-2, 2.0 * ev, 1.0 * fs, 2.0 * fs, 0.0, 1e30)
        g.add_source("x", 1e-2, 2.5 * ev, 1.0 * fs, 2.0 * fs, [(3 * q - n // 2) * dr], 4 * dr, 0.0, 1e30)
        g.add_plane_source(1, 1, 3 * q + 1, 1e-2, 3.0 * ev, 1.0 * fs, 2.0 * fs, 0.0, 0.5 * fs)
        groups = []
        r = np.random.default_rng(n + 1)
        for model, ne in ((1, 9), (2, 5)):
            cells = (3 * q + 2 + r.integers(0, 2 * q, ne))[:, None].astype(np.int32)
            cells[:2, 0] = 3 * q, 5 * q + 2
            par = [np.full((ne, model), 2.5 * ev), np.full((ne, model), 2.0), np.full((ne, 1), 4e4),
                   np.full((ne, 1), 4e3), r.uniform(0.2, 1.0, (ne, 3))]
            groups.append(g.add_q_group(omx.Q_MATERIAL, model, cells, np.concatenate(par, 1), 1e-4, skip * dt))
        for p in (2, 3 * q, 5 * q + 1, n - 1):
            g.add_detector(omx.POINT, "Ex", [[p]])
        f = np.zeros([h - b + 1 for b, h in zip(*g.field_bounds(1))], order="F")
        a0 = 1 - g.field_bounds(1)[0][0]
        f[a0 + 1:a0 + n - 1] = (1e-3 * np.random.default_rng(n).standard_normal(n - 2)).reshape((n - 2,) + f.shape[1:])
        g.write_field(1, f)
        for tt, k in ((1, 2), (3, 1), (4, 33)):
            g.run(tt, k, skip, 3, use_graph=graph)
        out.append([np.concatenate([v.ravel() for v in g.drain_detectors()])] + [g.read_field(x) for x in (1, 5)] +
                   [v for gr in groups for v in gr.read().values()])
        g.kill()
    assert all(np.max(np.abs(v)) > 0 for v in out[0][:3]) and np.max(np.abs(out[0][-1])) > 0
    for a, b in zip(*out):
        assert np.array_equal(a, b)


def test_closure_step_tiles():
    """The recurrent steps' column tiles by the number of rows (32, 64, 128 columns, chained or not):
    sequences do not interact, so each gives the same bits in every batch, and the gradient of a
    batch of 2^k copies is that of one copy: per-row terms scale by powers of two exactly, sums of
    49152 FP32 terms agree to about 1e-5 of their largest with cancellation of up to 100."""
    from test_gpu_closure import co

    params = co.init_params(3).astype(np.float32)
    cl = omx.Closure(params, 1.0, 1.0)
    rng = np.random.default_rng(3)
    T = 6
    e = rng.standard_normal((8, T + 31)).astype(np.float32)
    y = cl.forward(e, T)
    assert np.max(np.abs(y)) > 0
    for copies in (2, 144, 145, 304, 305, 4097): # the last and first rows of each forward tile width
        yy = cl.forward(np.tile(e, (copies, 1)), T).reshape(T, copies, 8)
        assert np.array_equal(yy, np.broadcast_to(np.asarray(y).reshape(T, 1, 8), yy.shape))
    tgt = rng.standard_normal((T, 8)).astype(np.float32)
    loss, g = cl.gradient(e, tgt, 1)
    for copies in (1024, 2048):                  # backward tiles of 64 and of 128 columns; one copy: 32
        l2, g2 = cl.gradient(np.tile(e, (copies, 1)), np.tile(tgt, (1, copies)), 1)
        assert abs(l2 - loss) <= 1e-9 * abs(loss)
        assert np.max(np.abs(g2 - g)) <= 1e-3 * np.max(np.abs(g))
    cl.kill()


@pytest.mark.parametrize("dims,n,precision,shape", [
    (1, (200,), "fp64", None), (2, (70, 60), "fp32", None), (2, (70, 60), "fp64", None),
    (3, (30, 26, 28), "fp32", None), (3, (30, 26, 28), "fp32", 8016), (3, (30, 26, 28), "fp64", None),
])
def test_prepared_run_equals_run(dims, n, precision, shape):
    """A run whose step graphs were captured beforehand steps through its table as any other."""
    dt = omx.units.yee_dt(37.8)
    out = []
    for prepared in (False, True):
        g = omx.TMxll(dims, n, 4, (3,) * 3, dt, 37.8, mode=omx.TMZ, precision=precision)
        comp = 3 if dims == 2 else 1
        g.add_plane_source(comp, dims, n[dims - 1] // 2, 1e-2, 0.1, 8 * dt, 6 * dt, 0.0, 1e30)
        g.add_detector(omx.POINT, "Ez" if dims == 2 else "Ex", [[m // 2 for m in n]])
        if shape:
            g.set_launch_shape(shape)
        g.run(1, 3, 1, 1)
        if prepared:
            g.prepare_run(4, 20, 1, 1)
        g.run(4, 20, 1, 1)
        out.append(list(g.drain_detectors()) + [g.read_field(comp)])
        g.kill()
    assert np.max(np.abs(out[0][1])) > 0
    for a, b in zip(*out):
        assert np.array_equal(a, b)


# what happens to member 0 between two odd-length runs of the batch: a staged shape or the two-pass form of
# its own, runs in a second (staged) batch, a source on dispersive cells (two half-step passes from
# then on, for every member)
@pytest.mark.parametrize("use_graph", [True, False])
@pytest.mark.parametrize("change", ["shape", "two_pass", "single_pass", "second", "source"])
def test_inplace_batch_after_its_members_change(change, use_graph):
    """A batch steps in its own form whatever happens to its members between runs: every member
    equals its solo run bit for bit, and a member's own form is its own afterwards."""
    from test_gpu_parity import fused3_deck
    from omx import decks

    specs = [((33, 30, 27), (3, 3, 3)), ((40, 36, 28), (3, 3, 2)), ((29, 41, 26), (1, 3, 3))]

    def build(spec):
        d = fused3_deck(*spec, src="both")
        g = omx.TMxll(3, d["grid_Ndims"], d["npml"], d["boundaries"], d["dt"], d["dr"], precision="fp32")
        gr = decks.apply_deck(g, d, omx, decks.media_map(d, omx.media_map_from_voxels))
        for det in d["detectors"]:
            g.add_detector(det["type"], det["field"], det["idx"])
        return g, gr

    def state(g, gr):
        return [g.drain_detectors()[1]] + [g.read_field(f) for f in range(1, 7)] + [q.read()["rho"] for q in gr]

    def add_source(g):
        fs = omx.UNITS["fs_to_au"]
        g.add_plane_source(1, 3, 27 // 2, 1.0, 0.08, 1.0 * fs, 1.0 * fs, 0.0, 1e30)

    want = []
    for q, sp in enumerate(specs):
        g, gr = build(sp)
        g.run(1, 13, 1, 1)
        if change == "source":
            add_source(g) if q == 0 else g.set_step_form(omx.STEP_TWO_PASS)
        if change == "second" and q == 0:
            g.run(14, 5, 1, 1)
        g.run(19, 7, 1, 1)
        want.append(state(g, gr))
        g.kill()
    grids = [build(sp) for sp in specs]
    b = omx.Batch([g for g, _ in grids])
    b.run(1, 13, 1, 1, use_graph=use_graph)
    m = grids[0][0]
    if change == "shape":
        m.set_launch_shape(8064)
    elif change == "two_pass":
        m.set_step_form(omx.STEP_TWO_PASS)
    elif change == "single_pass":
        m.set_step_form(omx.STEP_SINGLE_PASS)
    elif change == "source":
        add_source(m)
    else:
        b2 = omx.Batch([m])
        b2.set_launch_shape(8016)
        b2.run(14, 5, 1, 1, use_graph=use_graph)
        b2.synchronize()
        b2.kill()
    b.run(19, 7, 1, 1, use_graph=use_graph)
    b.synchronize()
    for (g, gr), w in zip(grids, want):
        got = state(g, gr)
        assert np.max(np.abs(w[0])) > 0
        for x, y in zip(got, w):
            assert np.array_equal(x, y)
    b.kill()
    for g, _ in grids:
        g.kill()


@pytest.mark.parametrize("staged", [False, True])
def test_batch_leaves_its_members_own_shape(staged):
    """A member that ran in a batch launches what a grid that did not launches afterwards."""
    def launches(batch):
        dt = omx.units.yee_dt(37.8)
        g = omx.TMxll(3, (30, 26, 28), 4, (3,) * 3, dt, 37.8, precision="fp32")
        if batch:
            b = omx.Batch([g])
            if staged:
                b.set_launch_shape(8016)
            b.run(1, 4)
            b.synchronize()
            b.kill()
        else:
            g.run(1, 4)
        n = g.launch_count()
        g.run(5, 6, use_graph=False)
        n = g.launch_count() - n, g.algorithmic_bytes(omx.KC_E)
        g.kill()
        return n

    assert launches(True) == launches(False)


@pytest.mark.parametrize("before", ["nothing", "shape", "autotune", "batch"])
def test_single_pass_form_is_the_staged_pass(before):
    """OMX_STEP_SINGLE_PASS steps 3D grids in the staged pass also after the passes in place were
    selected by a shape, by the tuner or by a batch; the default form returns to them."""
    dt = omx.units.yee_dt(37.8)
    g = omx.TMxll(3, (30, 26, 28), 4, (3,) * 3, dt, 37.8, precision="fp32")
    if before == "shape":
        g.set_launch_shape(4)
    elif before == "autotune":
        g.autotune(reps=1)
        g.set_launch_shape(2)                # whatever the tuner's pick
    elif before == "batch":
        b = omx.Batch([g])
        b.run(1, 2)
        b.synchronize()
        b.kill()
    words = {}
    for form in (omx.STEP_DEFAULT, omx.STEP_SINGLE_PASS, omx.STEP_DEFAULT):
        g.set_step_form(form)
        g.run(3, 3)
        words.setdefault(form, set()).add(g.algorithmic_bytes(omx.KC_E))
    g.kill()
    # 18 words a cell and step in place, 12 staged, beside the same CPML words
    (inplace,), (staged,) = words[omx.STEP_DEFAULT], words[omx.STEP_SINGLE_PASS]
    assert inplace - staged == 6 * 4 * 30 * 26 * 28


# a pass in place launches at most 65535 blocks along y and along z: (32, 4, 21846) and (30, 3, 21850) all
# dispersive have a list of more block layers than that (three entries a cell, 128 a block),
# (32, 4, 20000) one that leaves few layers to the planes, (3, 262145, 3) has too many rows
@pytest.mark.parametrize("n,media", [
    ((32, 4, 21846), "all"), ((30, 3, 21850), "all"), ((32, 4, 20000), "all"), ((4, 4, 70001), "none"),
    ((3, 262140, 3), "some"), ((3, 262145, 3), "some"),
])
def test_inplace_launches_of_long_thin_grids(n, media):
    """Launch limits of the 3D pass in place: fields as from the staged pass, bit for bit, at the default
    march and (where the rows fit) one plane a thread."""
    dr = 37.8
    dt = omx.units.yee_dt(dr)
    out = []
    for form, shape in ((omx.STEP_SINGLE_PASS, None), (omx.STEP_DEFAULT, None), (omx.STEP_DEFAULT, 1)):
        g = omx.TMxll(3, n, 4, (1, 1, 1), dt, dr, precision="fp32")
        if media != "none":
            m = np.zeros(n + (3,), np.int32, order="F")    # a medium per component
            m[tuple(slice(None) if media == "all" else slice(1, max(2, q // 2)) for q in n)] = 1
            g.set_media([omx.medium_drude(0.33, 0.01, 1.5, dt)], m)
        a = int(np.argmax(n))
        g.add_plane_source(3 if a != 2 else 1, a + 1, n[a] // 2, 1e-2, 0.1, 2 * dt, 3 * dt, 0.0, 1e30)
        g.set_step_form(form)
        if shape:
            g.set_launch_shape(shape)
        g.run(1, 6)
        out.append([g.read_field(f) for f in range(1, 7)])
        g.kill()
    assert max(np.max(np.abs(f)) for f in out[0]) > 0
    for o in out[1:]:
        for a, b in zip(o, out[0]):
            assert np.array_equal(a, b)


def test_fields_beyond_31_bit_offsets_step_in_two_passes():
    """A 3D grid whose fields have more words than the fused pass's 31-bit offsets reach takes the two
    half-step passes: a source beyond the limit radiates as in a small grid, bit for bit."""
    dr = 37.8
    dt = omx.units.yee_dt(dr)
    out = []
    for n, z in (((1300, 1300, 1280), 1262), ((64, 64, 64), 32)):
        g = omx.TMxll(3, n, 4, (1, 1, 1), dt, dr, precision="fp32")
        if n[0] > 64:
            for staged in (8064, 8016):
                with pytest.raises(omx.OMXError):
                    g.set_launch_shape(staged)
            g.set_launch_shape(4)            # planes per thread of the two passes
        else:
            g.set_step_form(omx.STEP_TWO_PASS)
        off = z - n[2] // 2
        g.add_source("z", 1e-2, 0.1, 2 * dt, 3 * dt, (0.0, 0.0, (off + 0.5) * dr if off else 0.0), 1.5 * dr, 0.0, 1e30)
        c = (n[0] // 2, n[1] // 2, z)
        for f in ("Ex", "Ey", "Ez", "Hx", "Hy", "Hz"):
            g.add_detector(omx.POINT, f, [[c[0] + a, c[1] + b, c[2] + k] for a, b, k in ((0, 0, 0), (2, 1, -2), (-3, 2, 3))])
        g.run(1, 9, 1, 1)
        out.append(g.drain_detectors()[1])
        g.kill()
    reached = np.max(np.abs(out[1]), axis=0).reshape(6, 3)
    assert np.all(reached[:, 1:] > 0)        # on the source's axis the transverse components vanish
    assert np.array_equal(*out)


def test_batch_tuners_choice_keeps_its_form():
    """omx_batch_set_launch_shape(omx_batch_autotune's choice) keeps the form that the tuner kept; another
    shape selects the staged pass.  Results as from an untuned batch, bit for bit."""
    dt = omx.units.yee_dt(37.8)

    def build():
        grids = [omx.TMxll(3, n, 4, (3,) * 3, dt, 37.8, precision="fp32") for n in ((30, 26, 28), (24, 33, 29))]
        for g in grids:
            g.add_plane_source(1, 3, 14, 1e-2, 0.1, 4 * dt, 5 * dt, 0.0, 1e30)
        return grids, omx.Batch(grids)

    grids, b = build()
    choice = b.autotune(reps=20)
    form = []
    for tt, shape in ((1, None), (6, choice), (11, 8016 if choice != 8016 else 8032), (16, choice)):
        if shape:
            b.set_launch_shape(shape)
        b.run(tt, 5)
        b.synchronize()
        form.append([g.algorithmic_bytes(omx.KC_E) for g in grids])
    assert form[0] == form[1] == form[3]
    cells = np.array([30 * 26 * 28, 24 * 33 * 29])
    assert np.all((np.array(form[0]) - form[2] == 24 * cells) | (np.array(form[0]) == form[2]))
    plain, b2 = build()
    b2.run(1, 20)
    b2.synchronize()
    for g, q in zip(grids, plain):
        for f in range(1, 7):
            assert np.array_equal(g.read_field(f), q.read_field(f))
    assert np.max(np.abs(plain[0].read_field(1))) > 0
    for x in (b, b2, *grids, *plain):
        x.kill()


@pytest.mark.parametrize("n,count,inplace", [(20, 48, True), (20, 49, False), (74, 49, True)])
def test_batch_form_by_number_and_size_of_members(n, count, inplace):
    """Many small grids step in the staged batch, few or larger ones in place; members equal solo runs."""
    dt = omx.units.yee_dt(37.8)

    def build(k):
        g = omx.TMxll(3, (n, n, n), 4, (3,) * 3, dt, 37.8, precision="fp32")
        g.add_plane_source(1, 3, n // 2, 1e-2 * (1 + k), 0.1, 4 * dt, 5 * dt, 0.0, 1e30)
        return g

    grids = [build(k) for k in range(count)]
    b = omx.Batch(grids)
    b.run(1, 9)
    b.synchronize()
    solo = build(count - 1)
    solo.set_step_form(omx.STEP_SINGLE_PASS)
    solo.run(1, 9)
    staged = solo.algorithmic_bytes(omx.KC_E)
    for g in (grids[0], grids[-1]):
        assert g.algorithmic_bytes(omx.KC_E) - staged == (24 * n ** 3 if inplace else 0)
    for f in range(1, 7):
        assert np.array_equal(grids[-1].read_field(f), solo.read_field(f))
    assert np.max(np.abs(solo.read_field(1))) > 0
    for x in (b, solo, *grids):
        x.kill()


# (8, 70001): more rows than a launch takes blocks along y
@pytest.mark.parametrize("n,precision,mode", [((243, 161), "fp32", 2), ((243, 161), "fp64", 1), ((8, 70001), "fp32", 2)])
def test_tuner_of_unfused_2d_grids(n, precision, mode):
    """The tuner looks at the short marches that the rule by size takes on small grids (a march of 8 rows
    takes such a grid twice as long); the tuned grid gives the untuned one's bits."""
    dt = omx.units.yee_dt(37.8)
    out = []
    for tuned in (False, True):
        g = omx.TMxll(2, n, 3, (2, 3, 1), dt, 37.8, mode=mode, precision=precision)
        comp = 3 if mode == 1 else 1
        g.add_plane_source(comp, 2, n[1] // 2, 1e-2, 0.1, 4 * dt, 5 * dt, 0.0, 1e30)
        if tuned:
            choice = g.autotune(reps=10)
            assert choice <= 4 if n[1] < 65536 else choice >= 2
        g.run(1, 12)
        out.append([g.read_field(f) for f in ((3, 4, 5) if mode == 1 else (1, 2, 6))])
        g.kill()
    assert np.max(np.abs(out[0][0])) > 0
    for a, b in zip(*out):
        assert np.array_equal(a, b)


# radial sources of one point, of a piece of the cells or less, over several pieces, from the first cell to
# the last, and of more points than the loop in one launch takes
@pytest.mark.parametrize("n,radii", [(200, (0, 30)), (1500, (16, 256, 400)), (6151, (2000, 16, 700, 1)),
                                     (401, (200,)), (6151, (1400, 1400, 1400))])
def test_one_launch_1d_loop_wide_sources(n, radii):
    """Radial 1D sources of any width in the loop in one launch: the bits of one launch per phase, and
    no slower than those (a thread looks at its own cells, not at every point)."""
    import time

    dr = 37.8
    dt = omx.units.yee_dt(dr)
    out, took = [], []
    for graph in (True, False):
        g = omx.TMxll(1, (n,), 5, (3, 1, 1), dt, dr, precision="fp64")
        for q, r in enumerate(radii):
            at = 0 if r >= n // 2 - 1 else (q - 1) * (n // 2 - r - 1) // 2
            g.add_source("x", 1e-2 * (q + 1), 0.1 + 0.03 * q, 5 * dt, 6 * dt, [(at + (0.5 if at >= 0 else -0.5)) * dr],
                         (r + 0.5) * dr, 0.0, 1e30)
        g.add_detector(omx.POINT, "Ex", [[n // 2]])
        g.run(1, 40, 1, 3, use_graph=graph)
        out.append([g.drain_detectors()[1]] + [g.read_field(f) for f in (1, 5)])
        t = []
        for k in range(5):
            g.synchronize()
            t0 = time.perf_counter()
            g.run(41 + 100 * k, 100, use_graph=graph)
            g.synchronize()
            t.append(time.perf_counter() - t0)
        took.append(min(t))
        g.kill()
    assert all(np.max(np.abs(v)) > 0 for v in out[0])
    for a, b in zip(*out):
        assert np.array_equal(a, b)
    assert took[0] < took[1]


@pytest.mark.parametrize("emitters,tuned,inplace", [(41723, False, True), (41724, False, False), (41724, True, False)])
def test_3d_form_by_emitters(emitters, tuned, inplace):
    """Emitters overlap less of the step in place: past emitters x cells^2 = 7e17 a grid takes the staged
    pass, tuned or not; both forms give the same bits."""
    n, dr = (160, 160, 160), 37.8
    ev, dt = omx.UNITS["ev_to_au"], omx.units.yee_dt(37.8)
    out, words = [], []
    for form in (omx.STEP_DEFAULT, omx.STEP_SINGLE_PASS):
        g = omx.TMxll(3, n, 4, (3,) * 3, dt, dr, precision="fp32")
        g.set_step_form(form)
        g.add_plane_source(1, 3, 80, 1e-2, 2.5 * ev, 2 * dt, 3 * dt, 0.0, 1e30)
        r = np.random.default_rng(1)
        cells = np.stack([r.integers(20, m - 20, emitters) for m in n], 1).astype(np.int32)
        par = [np.full((emitters, 1), 2.5 * ev), np.full((emitters, 1), 2.0), np.full((emitters, 1), 4e4),
               np.full((emitters, 1), 4e3), r.uniform(0.2, 1.0, (emitters, 3))]
        q = g.add_q_group(omx.Q_MATERIAL, omx.TWO_LEVEL, cells, np.concatenate(par, 1), 1e-5, dt)
        if tuned:
            g.autotune(reps=1)
        g.run(1, 7)
        words.append(g.algorithmic_bytes(omx.KC_E))
        out.append([g.read_field(f) for f in range(1, 7)] + [q.read()["rho"]])
        g.kill()
    assert words[0] - words[1] == (24 * 160 ** 3 if inplace else 0)
    assert np.max(np.abs(out[0][0])) > 0 and np.max(np.abs(out[0][-1])) > 0
    for a, b in zip(*out):
        assert np.array_equal(a, b)


# a launch with the dot products up to 256 cells, pieces of 128 cells past them
@pytest.mark.parametrize("n,n_der", [(100, 1), (1000, 2), (32640, 2), (32641, 3), (100003, 4)])
def test_fd_1d_operator(orc, n, n_der):
    """The 1D operator against the oracle, bit for bit, and at a cost a cell like the 2D operator's (each
    thread computes what it stores, once)."""
    rng = np.random.default_rng(n)
    eps = 1.0 + 1.25 * (rng.random(n) < 0.4) + 0.3j
    G = omx.FDOperator((n,), 4, n_der, (2,), 0.25, 1.3, eps)
    O = orc.FDOperator((n,), 4, n_der, (2,), 0.25, 1.3, eps)
    f = G.zeros()
    f[:, n_der:n_der + n] = rng.normal(size=(4, n)) + 1j * rng.normal(size=(4, n))
    own = (slice(None), slice(n_der, n_der + n))
    for transpose in (False, True):
        assert np.array_equal(G.apply(f, transpose)[own], O.apply(f, transpose)[own])
    if n > 10 ** 5:
        P = omx.FDOperator((400, 250), 4, n_der, (2, 2), 0.25, 1.3, np.ones((400, 250)))
        t1, t2 = (min(op.time_apply(20) for _ in range(3)) for op in (G, P))
        assert t1 < 2.0 * t2                 # 0.64 measured, 2.2 with every component in each component's thread
        P.kill()
    G.kill()


# padded arrays of at most 4096 words and groups of at most 2500 emitters are arranged on the host, larger
# ones on the device; ghost planes of periodic axes read as zero
@pytest.mark.parametrize("dims,n,bnd,emitters", [
    (1, (4079,), (3, 1, 1), 2500), (1, (4080,), (3, 1, 1), 2501), (1, (4063,), (3, 1, 1), 1), (2, (60, 62), (2, 3, 1), 7),
    (2, (60, 63), (3, 2, 1), 3000), (3, (11, 9, 20), (2, 3, 2), 40), (3, (27, 9, 30), (3, 2, 2), 400),
])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_reads_of_small_and_large_arrays(dims, n, bnd, emitters, precision):
    """Fields read as written, on both sides of the sizes where the way of reading changes, and emitters in
    the caller's order, each with the state that it has alone."""
    dr = 37.8
    ev, dt = omx.UNITS["ev_to_au"], omx.units.yee_dt(37.8)
    rng = np.random.default_rng(sum(n))
    g = omx.TMxll(dims, n, 2, bnd, dt, dr, mode=1, precision=precision)
    fields = {1: [1, 5], 2: [3, 4, 5], 3: [1, 2, 3, 4, 5, 6]}[dims]
    for f in fields:
        lo, hi = g.field_bounds(f)
        a = np.asfortranarray(rng.standard_normal([h - b + 1 for b, h in zip(lo, hi)]).astype(np.float32).astype(float))
        g.write_field(f, a)
        for x in range(dims):
            if f <= 3 and bnd[x] == 2 and hi[x] == n[x] + 1:
                a[(slice(None),) * x + (-1,)] = 0.0
        assert np.array_equal(g.read_field(f), a)
    cells = np.stack([rng.integers(2, m - 1, emitters) for m in n], 1).astype(np.int32)
    w = rng.uniform(1.0, 3.0, emitters) * ev
    par = np.stack([w, np.full(emitters, 2.0), np.full(emitters, 4e4), np.full(emitters, 4e3)], 1)
    q = g.add_q_group(omx.Q_MATERIAL, omx.TWO_LEVEL, cells,
                      np.concatenate([par, np.ones((emitters, 3))], 1), 1e-9, dt)
    g.q_group_step(q, 1)
    got = q.read()
    pick = sorted(set(rng.integers(0, emitters, 5)) | {0, emitters - 1})
    one = omx.TMxll(dims, n, 2, bnd, dt, dr, mode=1, precision=precision)
    for f in fields:
        one.write_field(f, g.read_field(f))
    alone = [one.add_q_group(omx.Q_MATERIAL, omx.TWO_LEVEL, cells[e:e + 1],
                             np.concatenate([par[e:e + 1], np.ones((1, 3))], 1), 1e-9, dt) for e in pick]
    for e, r in zip(pick, alone):
        one.q_group_step(r, 1)
        for k, v in r.read().items():
            assert np.array_equal(v[0], got[k][e]), (e, k)
    assert np.max(np.abs(got["E"])) > 0
    g.kill()
    one.kill()
