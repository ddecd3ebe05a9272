"""The work a user of this framework has it do, as cases to be measured.

A program that uses the framework admits runs, gives each its primitives, advances it by some steps
of the RK3 GRMHD update and reads the primitives back; a sweep or a server advances many small runs
together; a driver that keeps its own time loop asks for the fluxes alone.  The cases are these calls
over the grids of the benchmark, the tests and the serving stream.

kind    what a pass is
torus   a Fishbone-Moncrief torus (3D, or the axisymmetric phi slab where nph is 0): the primitives
        come from an array in GPU memory, the run takes `steps` steps and the primitives are read back
        into GPU memory (with host true: from and to pinned host memory, as a host code calls it)
tori    axisymmetric tori of several grids, spins and precisions advanced together (rg_step_batch),
        as the serving loop does between arrivals
tubes   seeded Riemann tubes of several lengths advanced together
calflx  the face fluxes of given primitives into the caller's buffer (rg_calflx_static)

`exact` restates the update in 64-bit torch operations (grid, metric, reconstruction, Lax-Friedrichs
fluxes, flux-CT, geometric source, RK3, the two Newton-Raphson inversions, ghost fills and floors).
"""
import math

import numpy as np
import torch

from raishinsource_b200 import Context, config

NAMES = ("rho", "u1", "u2", "u3", "p", "s", "b1", "b2", "b3")


# ---------------------------------------------------------------- the cases
def listed():
    return [
        # a 1D shock tube, the first run anybody tries: a handful of blocks, launches are all there is
        dict(name="tube_400", kind="tubes", lengths="400", copies=1, irec=6, precision="fp64", steps=4),
        # the smallest 3D torus of the tests: every kernel of a step on a nearly empty GPU
        dict(name="torus_40x24x16", kind="torus", nr=40, nth=24, nph=16, irec=6, precision="fp64", steps=4, host=False),
        # axisymmetric tori: the small one of the tests and the one of the benchmark
        dict(name="torus2d_64x64", kind="torus", nr=64, nth=64, nph=0, irec=6, precision="fp64", steps=8, host=False),
        dict(name="torus2d_256x256", kind="torus", nr=256, nth=256, nph=0, irec=6, precision="fp64", steps=8, host=False),
        # the serving mix: axisymmetric tori of every size and of both precisions in flight at once
        dict(name="serve_6", kind="tori", grids="128,256,384,512,256,128", irec=6, steps=4),
        # a parameter sweep of 1D tubes, 400 to 3200 cells each
        dict(name="tubes_64", kind="tubes", lengths="400,900,1801,3200", copies=16, irec=6, precision="fp64", steps=6),
        # an odd 3D grid (no extent a multiple of a tile) with WENO5
        dict(name="torus_131x61x47_weno5", kind="torus", nr=131, nth=61, nph=47, irec=7, precision="fp64", steps=1,
             host=False),
        # PPM, the scheme that needs no positivity fallback
        dict(name="torus_192x96x96_ppm", kind="torus", nr=192, nth=96, nph=96, irec=5, precision="fp64", steps=1, host=False),
        # the benchmark's torus, its arrays kept on the GPU, and called from a host code
        dict(name="torus_256x128x128", kind="torus", nr=256, nth=128, nph=128, irec=6, precision="fp64", steps=1, host=False),
        dict(name="host_256x128x128", kind="torus", nr=256, nth=128, nph=128, irec=6, precision="fp64", steps=1, host=True),
        # the largest grid of the benchmark, FP32 beyond twice the horizon radius
        dict(name="torus_384x192x192_mixed", kind="torus", nr=384, nth=192, nph=192, irec=6, precision="mixed", steps=1,
             host=False),
        # the fluxes alone, for a driver with its own update
        dict(name="calflx_64x64x64", kind="calflx", nr=64, nth=64, nph=64, irec=6),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["torus3d", "torus3d", "torus2d", "tori", "tubes", "calflx"])
    irec = rng.choice([6, 6, 5, 7])
    if kind == "torus3d":
        host = rng.random() < 0.2
        top = 128 if irec != 6 or host else 176
        nr, nth, nph = _log_int(rng, 40, 2 * top), _log_int(rng, 24, top), _log_int(rng, 16, top)
        prec = "mixed" if rng.random() < 0.3 else "fp64"
        return dict(kind="torus", nr=nr, nth=nth, nph=nph, irec=irec, precision=prec, steps=1, host=host)
    if kind == "torus2d":
        prec = rng.choice(["fp64", "mixed"])
        return dict(kind="torus", nr=_log_int(rng, 48, 512), nth=_log_int(rng, 48, 512), nph=0, irec=irec, precision=prec,
                    steps=rng.randint(2, 8), host=False)
    if kind == "tori":
        grids = ",".join(str(_log_int(rng, 96, 512)) for _ in range(rng.randint(2, 8)))
        return dict(kind="tori", grids=grids, irec=6, steps=rng.randint(2, 4))
    if kind == "tubes":
        lengths = ",".join(str(_log_int(rng, 400, 3200)) for _ in range(rng.randint(1, 4)))
        return dict(kind="tubes", lengths=lengths, copies=rng.randint(1, 24), irec=6,
                    precision=rng.choice(["fp64", "mixed"]), steps=rng.randint(2, 6))
    # at most 262144 cells, the call's limit
    nr, nth = _log_int(rng, 40, 128), _log_int(rng, 24, 64)
    return dict(kind="calflx", nr=nr, nth=nth, nph=max(16, min(64, 262144 // (nr * nth) - 1)), irec=irec)


def _grids(case):
    """The parameter blocks of a case's runs."""
    if case["kind"] == "tubes":
        return [dict(config.tube(n=int(n), irec=case["irec"], precision=case["precision"]), guard=1)
                for n in case["lengths"].split(",") for _ in range(case["copies"])]
    if case["kind"] == "tori":
        return [dict(config.torus(nr=int(g), nth=int(g), irec=case["irec"], akm=(0.0, 0.5, 0.9375)[k % 3],
                                  precision=("fp64", "mixed")[k % 2]), guard=1)
                for k, g in enumerate(case["grids"].split(","))]
    return [dict(config.torus(nr=case["nr"], nth=case["nth"], nph=case["nph"] or None, irec=case["irec"],
                              precision=case.get("precision", "fp64")), guard=1)]


# ------------------------------------------------------- prepare, run, work
_context = None


def _ctx():
    global _context
    if _context is None:
        _context = Context(0)
    return _context


class _State:
    """The admitted runs of a case and the arrays a program hands over with them."""

    def __init__(self, case, runs, arrays):
        self.case, self.runs, self.arrays = case, runs, arrays
        # a host code keeps its own result array; one on the GPU takes it from torch's pool
        self.out = _array(runs[0].params, True) if case.get("host") else None

    def __del__(self):
        for r in self.runs:
            r.release()


def _array(p, host=False):
    shape = (p["kmax"], p["jmax"], p["imax"], 9)
    return torch.empty(shape, dtype=torch.float64, pin_memory=True) if host else torch.empty(
        shape, dtype=torch.float64, device="cuda")


def prepare(case, seed):
    ctx = _ctx()
    runs, arrays = [], []
    for k, p in enumerate(_grids(case)):
        r = ctx.admit(p)
        runs.append(r)
        if case["kind"] == "tubes":
            r.ic_tube(seed=seed, tube=k)
        else:
            r.ic_torus_device(seed=seed + k, beta=100.0, rmax=12.0)
        a = _array(p, case.get("host", False))
        r.download_prims_ptr(a.data_ptr())
        if case["kind"] == "calflx":
            a = a.reshape(-1, 9).t().contiguous()
        arrays.append(a)
    torch.cuda.synchronize()
    return _State(case, runs, arrays)


def run(state):
    case, ctx = state.case, _ctx()
    if case["kind"] == "calflx":
        n = state.arrays[0].shape[1]
        ww = torch.empty(27, n, dtype=torch.float64, device="cuda")
        state.runs[0].calflx_static(state.arrays[0].data_ptr(), ww.data_ptr())
        return _interior_fluxes(ww, state.runs[0])
    if len(state.runs) == 1:
        out = _array(state.runs[0].params) if state.out is None else state.out
        outs = [out]
    else:  # the batch's results one after another in one array
        sizes = [a.numel() // 9 for a in state.arrays]
        out = torch.empty(sum(sizes), 9, dtype=torch.float64, device="cuda")
        outs = out.split(sizes)
    for r, a in zip(state.runs, state.arrays):
        r.upload_prims_ptr(a.data_ptr())
    if len(state.runs) == 1:
        state.runs[0].step(case["steps"])
    else:
        ctx.step_batch(state.runs, case["steps"])
    for r, o in zip(state.runs, outs):
        r.download_prims_ptr(o.data_ptr())
    return {n: out[..., v] for v, n in enumerate(NAMES)}


def _by_variable(outs):
    """{variable: tensor}; the runs of a batch one after another."""
    if len(outs) == 1:
        return {n: outs[0][..., v] for v, n in enumerate(NAMES)}
    return {n: torch.cat([o[..., v].reshape(-1) for o in outs]) for v, n in enumerate(NAMES)}


def _interior_fluxes(ww, r):
    """The fluxes on the faces the update of an interior cell reads (elsewhere the buffer is not written)."""
    kk, jj, ii, _ = r.shape
    w = ww.view(3, 9, kk, jj, ii)
    m = r.nm1 - 1
    return {"f%d_%s" % (d + 1, n): w[d, v, m:kk - m - 1, m:jj - m - 1, m:ii - m - 1]
            for d in range(3) for v, n in enumerate(NAMES)}


# FP64 operations of one zone and step (three stages: reconstruction and the
# two states of each face, flux-CT, source, RK combine, inversion, floors; one
# CFL reduction), counted on MP5: adds and multiplies, a fused one as two.
FLOPS_PER_ZONE_STEP = 15271.0


def work(case):
    total_b, total_f = 0.0, 0.0
    for p in _grids(case):
        n = p["imax"] * p["jmax"] * p["kmax"]
        z = config.interior_cells(p)
        geo = 142 * 8 * p["imax"] * p["kmax"]  # metric caches and Christoffel symbols, read once
        if case["kind"] == "calflx":
            total_b += 8 * (9 + 27) * n + 3 * 26 * 8 * p["imax"] * p["kmax"]
            total_f += z * 3400.0
            continue
        # primitives in and out in the reference layout, then the state once in and out per step
        total_b += 2 * 72 * n + case["steps"] * (2 * 72 * z + geo)
        total_f += case["steps"] * z * FLOPS_PER_ZONE_STEP
    return {"bytes": total_b, "flops": total_f}


def tolerance(case):
    # Measured against `exact`, whose operations are rounded in another order, over the listed cases and twelve
    # drawn ones, times four or more: the largest differences are those of u3, the small velocity across the
    # midplane (1.4e-11 in FP64, 1.4e-5 where FP32 faces, flux-CT and RK increments enter), and of the mass and
    # momentum fluxes (8.6e-11).
    if case["kind"] == "tori" or case.get("precision") == "mixed":
        return {"rel": 6e-5, "max": 3e-3}
    return {"rel": 4e-10, "max": 2e-8}


# --------------------------------------------------------------- 64-bit torch
PI = 3.14159265358979323


def _axis(n, lo, hi, kind, which):
    """Centres, face positions, their logical coordinates and the spacings dxb of one direction (1-based, index 0 unused)."""
    x, xb = np.zeros(n + 2), np.zeros(n + 2)
    i = np.arange(1, n + 1)
    if kind == 1:
        x[1:n + 1] = lo + (hi - lo) / (n - 1) * (i - 1)
        xb[:] = x
    elif which == "r":
        s0, s1 = math.log(lo), math.log(hi)
        xb[1:n + 1] = s0 + (i - 1) * ((s1 - s0) * float(np.float32(1.0) / np.float32(n - 1)))
        x[1:n + 1] = np.exp(xb[1:n + 1])
    else:
        t0, t1 = lo / PI, hi / PI
        xb[1:n + 1] = PI * (t0 + (i - 1) * ((t1 - t0) / (n - 1)))
        x[1:n + 1] = xb[1:n + 1] + 0.25 * np.sin(2 * xb[1:n + 1])  # hslope 0.5
    last_x = x[n] - x[n - 1] if kind == 1 else xb[n] - xb[n - 1]
    xa, xab = np.zeros(n + 2), np.zeros(n + 2)
    xa[1:n], xab[1:n] = 0.5 * (x[1:n] + x[2:n + 1]), 0.5 * (xb[1:n] + xb[2:n + 1])
    xa[n], xab[n] = xa[n - 1] + last_x, xab[n - 1] + last_x
    dxb = np.zeros(n + 2)
    dxb[2:n + 1] = xab[2:n + 1] - xab[1:n] if kind != 1 else xa[2:n + 1] - xa[1:n]
    dxb[1] = dxb[2]
    return x, xa, xb, dxb


def _kerr(a, r, th, thm):
    """Covariant modified Kerr-Schild metric on broadcast (theta, r) points."""
    r, th, thm = np.broadcast_arrays(r, th, thm)
    s2, c = np.sin(th) ** 2, np.cos(th)
    sig = r * r + a * a * c * c
    aa = (r * r + a * a) ** 2 - a * a * (r * r - 2 * r + a * a) * s2
    h = 1 + 0.5 * np.cos(2 * thm)
    g = np.zeros(r.shape + (4, 4))
    z = 2 * r / sig
    g[..., 0, 0] = -1 + z
    g[..., 0, 1] = g[..., 1, 0] = z * r
    g[..., 0, 2] = g[..., 2, 0] = -a * s2 * z
    g[..., 1, 1] = (1 + z) * r * r
    g[..., 1, 2] = g[..., 2, 1] = -a * s2 * (1 + z) * r
    g[..., 2, 2] = aa * s2 / sig
    g[..., 3, 3] = sig * h * h
    return g


class _Metric:
    def __init__(self, g, dev):
        gc = np.linalg.inv(g)
        t = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)[:, None, :]  # noqa: E731  (k, 1, i)
        self.g = [[t(g[..., m, n]) for n in range(4)] for m in range(4)]
        self.c = [[t(gc[..., m, n]) for n in range(4)] for m in range(4)]
        self.detg = t(np.sqrt(-np.linalg.det(g)))
        self.al = 1 / torch.sqrt(-self.c[0][0])
        self.be = [None] + [self.al ** 2 * self.c[0][m] for m in (1, 2, 3)]
        self.g3 = [None] + [self.c[m][m] + (self.be[m] / self.al) ** 2 for m in (1, 2, 3)]


class _Exact:
    """One run (or, for tubes of one length, several side by side along the second axis) in 64-bit torch.
    Arrays are [k, j, i]; a slab direction holds one plane."""

    def __init__(self, p, dev="cuda"):
        self.p, self.dev = p, dev
        self.nm0, self.nm1 = config.ghost_widths(p["irec"])
        self.mink = p["metric"] == 1
        nm1 = self.nm1
        self.jslab = p["jmax"] == 2 * nm1 + 1
        self.n = (p["imax"], p["jmax"], p["kmax"])
        ax = [_axis(p["imax"], p["xmin"], p["xmax"], p["ix1"], "r"), _axis(p["jmax"], p["ymin"], p["ymax"], 1, "phi"),
              _axis(p["kmax"], p["zmin"], p["zmax"], p["ix3"], "th")]
        self.slab = [False, self.jslab, self.mink]  # by direction r, phi, theta
        if self.mink:
            g = np.zeros((1, p["imax"], 4, 4))
            g[:] = np.diag([-1.0, 1.0, 1.0, 1.0])
            self.met = [None] + [_Metric(g, dev)] * 3
            self.chr = None
        else:
            (x1, x1a, x1b, _), (x3, x3a, x3b, _) = ax[0], ax[2]
            r, ra, s = x1[None, 1:-1], x1a[None, 1:-1], x1b[None, 1:-1]
            th, tha, thm = x3[1:-1, None], x3a[1:-1, None], x3b[1:-1, None]
            a = p["akm"]
            gc = _kerr(a, r, th, thm)
            self.met = [None, _Metric(_kerr(a, ra, th, thm), dev), _Metric(gc, dev), _Metric(_kerr(a, r, tha, thm), dev)]
            # Christoffel symbols by central differences of 1e-5 in the logical coordinates
            d, sm = 1e-5, 1e-12
            tp, tm = thm + d, thm - d
            dg = np.zeros(gc.shape + (4,))
            dg[..., 1] = (_kerr(a, np.exp(s + d), th, thm) - _kerr(a, np.exp(s - d), th, thm)) / (
                (s + d) - (s - d) + sm)[..., None, None]
            dg[..., 3] = (_kerr(a, r, tp + 0.25 * np.sin(2 * tp), tp) - _kerr(a, r, tm + 0.25 * np.sin(2 * tm), tm)) / (
                tp - tm + sm)[..., None, None]
            low = 0.5 * (np.einsum("...mln->...lmn", dg) + np.einsum("...nlm->...lmn", dg) - np.einsum("...nml->...lmn", dg))
            ch = np.einsum("...la,...amn->...lmn", np.linalg.inv(gc), low)
            self.chr = torch.from_numpy(ch).to(dev)[:, None]  # [k, 1, i, l, m, n]
        self.mc = self.met[2]
        f = lambda v: torch.from_numpy(np.array(v[1:-1])).to(dev)  # noqa: E731
        self.xs = [None, f(ax[0][0])[None, None, :], f(ax[1][0])[None, :, None], f(ax[2][0])[:, None, None]]
        self.dx = [None, f(ax[0][3])[None, None, :], f(ax[1][3])[None, :, None], f(ax[2][3])[:, None, None]]
        for d in (2, 3):
            if self.slab[d - 1]:
                dim = 3 - d
                self.dx[d] = self.dx[d].narrow(dim, nm1, 1)
                self.xs[d] = self.xs[d].narrow(dim, nm1, 1)
        rr = self.xs[1]
        self.fde, self.fpr = p["dmin"] * rr ** -1.5, (p["gam"] - 1) * p["pmin"] * rr ** -2.5

    def sh(self, a, dim, o):
        """a at the neighbour `o` cells up along dim (a slab direction is its own neighbour); wraps at the ends,
        where nothing reads it."""
        return a if o == 0 or self.slab[2 - dim] else torch.roll(a, -o, dim)

    # --- state algebra
    def qf(self, m, x):
        return (m.g[1][1] * x[1] * x[1] + 2 * m.g[1][2] * x[1] * x[2] + m.g[2][2] * x[2] * x[2] + m.g[3][3] * x[3] * x[3])

    def lower(self, m, v):
        return [m.g[0][0] * v[0] + m.g[0][1] * v[1] + m.g[0][2] * v[2], m.g[0][1] * v[0] + m.g[1][1] * v[1] + m.g[1][2] * v[2],
                m.g[0][2] * v[0] + m.g[1][2] * v[1] + m.g[2][2] * v[2], m.g[3][3] * v[3]]

    def upper(self, m, v):
        return [m.c[0][0] * v[0] + m.c[0][1] * v[1] + m.c[0][2] * v[2], m.c[1][0] * v[0] + m.c[1][1] * v[1] + m.c[1][2] * v[2],
                m.c[2][0] * v[0] + m.c[2][1] * v[1] + m.c[2][2] * v[2], m.c[3][3] * v[3]]

    def gfl(self, m, u):
        s = self.qf(m, [None] + u)
        s = torch.where(s < 0, torch.where(s.abs() <= 1e-10, s.abs(), torch.full_like(s, 1e-10)), s)
        s = torch.where(s.abs() > 5e2, torch.full_like(s, 5e2), s)
        return torch.sqrt(1 + s)

    def state(self, q, m):
        gam = self.p["gam"]
        S = {"q": q, "de": q[0], "pr": q[4], "gfl": self.gfl(m, [q[1], q[2], q[3]])}
        S["roh"] = q[0] + gam / (gam - 1) * q[4]
        b = [None, q[6], q[7], q[8]]
        ial = 1 / m.al
        uc = [S["gfl"] * ial] + [q[k] - S["gfl"] * m.be[k] * ial for k in (1, 2)] + [q[3]]
        ul = self.lower(m, uc)
        b0 = b[1] * ul[1] + b[2] * ul[2] + b[3] * ul[3]
        bc = [b0] + [(b[k] + b0 * uc[k]) / uc[0] for k in (1, 2, 3)]
        bl = self.lower(m, bc)
        S.update(uc=uc, ul=ul, bc=bc, bl=bl, b=b, bsq=sum(bc[k] * bl[k] for k in range(4)), sr=q[4] / q[0] ** gam)
        return S

    def cons(self, S, m):
        a, bb = S["roh"] + S["bsq"], S["pr"] + 0.5 * S["bsq"]
        uc, ul, bc, bl = S["uc"], S["ul"], S["bc"], S["bl"]
        u = [S["de"] * uc[0]] + [a * uc[0] * ul[k] - bc[0] * bl[k] for k in (1, 2, 3)]
        u += [a * uc[0] * ul[0] + bb - bc[0] * bl[0] + S["de"] * uc[0], S["de"] * S["sr"] * uc[0]] + S["b"][1:]
        return [m.detg * x for x in u]

    def flux(self, S, m, D):
        a, bb = S["roh"] + S["bsq"], S["pr"] + 0.5 * S["bsq"]
        uc, ul, bc, bl, b = S["uc"], S["ul"], S["bc"], S["bl"], S["b"]
        ud = uc[D]
        w = [S["de"] * ud] + [a * ud * ul[k] + (bb if k == D else 0.0) - bc[D] * bl[k] for k in (1, 2, 3)]
        w += [a * ud * ul[0] - bc[D] * bl[0] + S["de"] * ud, S["de"] * S["sr"] * ud]
        w += [torch.zeros_like(ud) if k == D else (ud / uc[0]) * b[k] - (uc[k] / uc[0]) * b[D] for k in (1, 2, 3)]
        return [m.detg * x for x in w]

    def speed(self, S, m, D):
        gam, q = self.p["gam"], S["q"]
        v = [None] + [q[k] / S["gfl"] for k in (1, 2, 3)]
        vsq = self.qf(m, v)
        cs, va = gam * S["pr"] / S["roh"], S["bsq"] / (S["roh"] + S["bsq"])
        om = va + cs * (1 - va)
        f1, f2 = v[D] * (1 - om), 1 - vsq * om
        f3 = torch.sqrt(om * (1 - vsq) * (f2 * m.g3[D] - (1 - om) * v[D] * v[D]))
        vp, vm = m.al * ((f1 + f3) / f2) - m.be[D], m.al * ((f1 - f3) / f2) - m.be[D]
        return torch.where(vp.abs() > 1, torch.ones_like(vp), vp), torch.where(vm.abs() > 1, -torch.ones_like(vm), vm)

    # --- reconstruction: the states of one cell at its upper and lower face along dim
    def mp5(self, u, dim):
        s = {o: self.sh(u, dim, o) for o in range(-2, 3)}
        sgn = lambda x: torch.copysign(torch.ones_like(x), x)  # noqa: E731
        mm = lambda x, y: 0.5 * (sgn(x) + sgn(y)) * torch.minimum(x.abs(), y.abs())  # noqa: E731

        def m4(w, x, y, z):
            k = torch.minimum(torch.minimum(w.abs(), x.abs()), torch.minimum(y.abs(), z.abs()))
            return 0.125 * (sgn(w) + sgn(x)) * (sgn(w) + sgn(y)).abs() * (sgn(w) + sgn(z)) * k

        d0, dm, dp = s[-1] - 2 * s[0] + s[1], s[-2] - 2 * s[-1] + s[0], s[0] - 2 * s[1] + s[2]
        out = []
        for sg in (1, -1):
            a2, a1, u0, b1, b2 = s[-2 * sg], s[-sg], s[0], s[sg], s[2 * sg]
            di, dl, dr = d0, (dm if sg > 0 else dp), (dp if sg > 0 else dm)
            ul = (2 * a2 - 13 * a1 + 47 * u0 + 27 * b1 - 3 * b2) / 60.0
            ump = u0 + mm(b1 - u0, 4 * (u0 - a1))
            d4p, d4m = m4(4 * di - dr, 4 * dr - di, di, dr), m4(4 * di - dl, 4 * dl - di, di, dl)
            uu, md = u0 + 4 * (u0 - a1), 0.5 * (u0 + b1) - sg * 0.5 * d4p
            lc = u0 + 0.5 * (u0 - a1) + sg * (4.0 / 3.0) * d4m
            lo = torch.maximum(torch.minimum(torch.minimum(u0, b1), md), torch.minimum(torch.minimum(u0, uu), lc))
            hi = torch.minimum(torch.maximum(torch.maximum(u0, b1), md), torch.maximum(torch.maximum(u0, uu), lc))
            out.append(torch.where((ul - u0) * (ul - ump) <= 1e-10, ul, ul + mm(hi - ul, lo - ul)))
        return out

    def weno5(self, u, dim):
        s = {o: self.sh(u, dim, o) for o in range(-2, 3)}
        c = float(np.float32(13.0) / np.float32(12.0))
        out = []
        for sg in (1, -1):
            a2, a1, u0, b1, b2 = s[-2 * sg], s[-sg], s[0], s[sg], s[2 * sg]
            e0 = c * (a2 - 2 * a1 + u0) ** 2 + 0.25 * (a2 - 4 * a1 + 3 * u0) ** 2 + 1e-6
            e1 = c * (a1 - 2 * u0 + b1) ** 2 + 0.25 * (a1 - b1) ** 2 + 1e-6
            e2 = c * (u0 - 2 * b1 + b2) ** 2 + 0.25 * (3 * u0 - 4 * b1 + b2) ** 2 + 1e-6
            w0, w1, w2 = 0.1 / e0 ** 2, 0.6 / e1 ** 2, 0.3 / e2 ** 2
            out.append((w0 * (2 * a2 - 7 * a1 + 11 * u0) + w1 * (-a1 + 5 * u0 + 2 * b1) + w2 * (2 * u0 + 5 * b1 - b2)) / (
                6 * (w0 + w1 + w2)))
        return out

    def ppm(self, q, D):
        dim = 3 - D
        dx = {o: self.sh(self.dx[D], dim, o - 1) for o in range(-4, 5)}  # the reference's spacing, one cell back
        xx = {o: self.sh(self.xs[D], dim, o) for o in (-1, 0, 1)}
        if self.slab[D - 1]:  # one plane: its neighbours' coordinates follow from the spacing
            xx = {o: self.xs[D] + o * self.dx[D] for o in (-1, 0, 1)}
        U = lambda v, o: self.sh(q[v], dim, o)  # noqa: E731
        one = torch.ones_like(q[0])
        zero = torch.zeros_like(one)

        def dda(o):
            return ((U(0, o + 1) - U(0, o)) / (dx[o + 1] + dx[o]) - (U(0, o) - U(0, o - 1)) / (dx[o] + dx[o - 1])) / (
                dx[o - 1] + dx[o] + dx[o + 1])

        ddp, ddm, rp, rm = dda(1), dda(-1), U(0, 1), U(0, -1)
        flat = (ddp * ddm >= 0) & ((rp - rm).abs() - 0.1 * torch.minimum(rp.abs(), rm.abs()) <= 0)
        et = -(ddp - ddm) / (xx[1] - xx[-1]) * (((xx[0] - xx[-1]) ** 3 + (xx[1] - xx[0]) ** 3) / (rp - rm))
        et = torch.where(flat, zero, et)
        eta = torch.clamp(torch.minimum(5 * (et - 0.05), one), min=0)
        pp, pm = U(4, 1), U(4, -1)
        weak = self.p["gam"] * ((rp - rm).abs() / torch.minimum(rp, rm)) < (pp - pm).abs() / torch.minimum(pp, pm)
        eta = torch.where(weak, zero, eta)

        def f1a(o):
            a, b = U(4, o + 1), U(4, o - 1)
            t3 = (a - b).abs()
            on = (torch.minimum(a, b) - t3 < 0) & (U(D, o + 1) - U(D, o - 1) < 0)
            t3b = U(4, o + 2) - U(4, o - 2)
            t4 = torch.where(t3b == 0, torch.where(t3 == 0, zero - 0.52, zero + 0.48), t3 / t3b - 0.52)
            return torch.minimum(one, torch.where(on, torch.clamp(10 * t4, min=0), zero))

        fl = torch.maximum(f1a(0), torch.where(pp - pm < 0, f1a(1), f1a(-1)))

        def dma(v, o):
            a, b, c = U(v, o - 1), U(v, o), U(v, o + 1)
            da = dx[o] / (dx[o - 1] + dx[o] + dx[o + 1]) * ((2 * dx[o - 1] + dx[o]) / (dx[o + 1] + dx[o]) * (c - b) + (
                dx[o] + 2 * dx[o + 1]) / (dx[o - 1] + dx[o]) * (b - a))
            k = torch.minimum((b - a).abs(), (c - b).abs()) * (1 if D == 3 else 2)
            return torch.where((c - b) * (b - a) <= 0, zero, torch.copysign(torch.minimum(da.abs(), k), da))

        def face(v, o, d0, d1):
            a, b, c, e = dx[o - 1], dx[o], dx[o + 1], dx[o + 2]
            u0, u1, t = U(v, o), U(v, o + 1), 1 / (dx[o - 1] + dx[o] + dx[o + 1] + dx[o + 2])
            t3 = t * (2 * c * b / (b + c)) * ((a + b) / (2 * b + c) - (e + c) / (2 * c + b))
            return u0 + b / (b + c) * (u1 - u0) + t3 * (u1 - u0) - t * b * (a + b) / (2 * b + c) * d1 + t * c * (
                c + e) / (b + 2 * c) * d0

        up, lo = [], []
        for v in range(9):
            dm, d0, dp, u0 = dma(v, -1), dma(v, 0), dma(v, 1), q[v]
            l, r = face(v, -1, dm, d0), face(v, 0, d0, dp)
            if v == 0:
                r = r * (1 - eta) + (U(v, 1) - 0.5 * dp) * eta
                l = l * (1 - eta) + (U(v, -1) + 0.5 * dm) * eta
            r, l = u0 * fl + r * (1 - fl), u0 * fl + l * (1 - fl)
            ext = (r - u0) * (l - u0) >= 0
            r, l = torch.where(ext, u0, r), torch.where(ext, u0, l)
            t3, t4 = 6 * (r - l) * (u0 - 0.5 * (r + l)), (r - l) ** 2
            l = torch.where(t3 > t4, 3 * u0 - 2 * r, l)
            r = torch.where(-t3 > t4, 3 * u0 - 2 * l, r)
            up.append(r)
            lo.append(l)
        return up, lo

    def faces(self, q, D):
        """Lax-Friedrichs fluxes of the faces above each cell along D."""
        dim, irec, m = 3 - D, self.p["irec"], self.met[D]
        if irec == 5:
            up, lo = self.ppm(q, D)
        else:
            both = [(self.mp5 if irec == 6 else self.weno5)(q[v], dim) for v in range(9)]
            up, lo = [b[0] for b in both], [b[1] for b in both]
        bad = lambda s: ~((s[0] > 0) & (s[4] > 0))  # noqa: E731
        ok, ol = bad(up), bad(lo)
        L = [torch.where(ok, q[v], up[v]) for v in range(9)]
        R = [self.sh(torch.where(ol, q[v], lo[v]), dim, 1) for v in range(9)]
        SL, SR = self.state(L, m), self.state(R, m)
        (vpL, vmL), (vpR, vmR) = self.speed(SL, m, D), self.speed(SR, m, D)
        z = torch.zeros_like(vpL)
        cx = torch.maximum(torch.maximum(z, vpR), vpL)
        cn = torch.minimum(torch.minimum(z, vpR if D == 3 else vmR), vmL)
        c1 = torch.maximum(cx.abs(), cn.abs())
        uL, uR, wL, wR = self.cons(SL, m), self.cons(SR, m), self.flux(SL, m, D), self.flux(SR, m, D)
        return [torch.where(cn > 0, wL[v], torch.where(cx > 0, 0.5 * (wL[v] + wR[v] - c1 * (uR[v] - uL[v])), wR[v]))
                for v in range(9)]

    def fluxes(self, q):
        """(F1, F2, F3) with flux-CT's six averaged induction fluxes in place."""
        F = [None] + [self.faces(q, d) for d in (1, 2, 3)]
        I, J, K = 2, 1, 0

        def avg(f, along, g, gm, gp):
            # (2 f + f(+along) + f(-along) - g - g(+gp) - g(-along) - g(-along, +gp)) / 8
            h = self.sh(g, along, -1)
            return (2 * f + self.sh(f, along, 1) + self.sh(f, along, -1) - g - self.sh(g, gp, 1) - h - self.sh(h, gp, 1)) / 8.0

        yx, zx, xy, zy, xz, yz = F[2][6], F[3][6], F[1][7], F[3][7], F[1][8], F[2][8]
        F[2][6], F[3][6] = avg(yx, I, xy, I, J), avg(zx, I, xz, I, K)
        F[1][7], F[3][7] = avg(xy, J, yx, J, I), avg(zy, J, yz, J, K)
        F[1][8], F[2][8] = avg(xz, K, zx, K, I), avg(yz, K, zy, K, J)
        return F

    # --- the update
    def interior(self):
        K, J, I = self.shape
        mask = torch.zeros(self.shape, dtype=torch.bool, device=self.dev)
        n = self.nm1
        mask[(slice(None) if K == 1 else slice(n, K - n)), (slice(None) if self.slab[1] else slice(n, J - n)), n:I - n] = True
        return mask

    def dt_of(self, q):
        S = self.state(q, self.mc)
        lim = 3 * self.nm1 - 1
        best = torch.ones_like(q[0])
        for D in (1, 2, 3):
            if self.n[D - 1] <= lim:
                continue
            vp, vm = self.speed(S, self.mc, D)
            v = torch.clamp(torch.maximum(vp.abs(), vm.abs()), max=1.0)
            best = torch.minimum(best, torch.where(v > 0, self.dx[D] / (v + 1e-12), torch.full_like(v, 1e10)))
        K, J, I = self.shape
        best = best[(slice(None) if K == 1 else slice(1, K - 1)), (slice(None) if self.slab[1] else slice(1, J - 1)), 1:I - 1]
        return self.p["cfl"] * best.amin(dim=(0, 2) if self.mink else (0, 1, 2), keepdim=True)

    def source(self, q):
        if self.chr is None:
            return [0.0] * 4
        S = self.state(q, self.mc)
        a, b = S["roh"] + S["bsq"], S["pr"] + 0.5 * S["bsq"]
        sf = [0.0] * 4
        for n in range(4):
            for m in range(4):
                t = a * S["uc"][m] * S["ul"][n] - S["bc"][m] * S["bl"][n]
                if m == n:
                    t = t + b
                for nu in range(4):
                    sf[nu] = sf[nu] + t * self.chr[..., n, nu, m]
        return [self.mc.detg * sf[nu] for nu in (1, 2, 3, 0)]

    def invert(self, u, qo, mask):
        """Primitives of the conserved u on mask (previous primitives qo), else qo."""
        at = mask.nonzero(as_tuple=True)
        pick = lambda a: a.expand(self.shape)[at]  # noqa: E731
        out = [x.clone() for x in qo]
        m = self.mc
        mm = _Metric.__new__(_Metric)
        mm.g = [[pick(x) for x in r] for r in m.g]
        mm.c = [[pick(x) for x in r] for r in m.c]
        mm.detg, mm.al = pick(m.detg), pick(m.al)
        got = self._invert([pick(x) for x in u], [pick(x) for x in qo], mm, at)
        for v in range(9):
            out[v][at] = got[v]
        return out

    def _invert(self, u, q, m, at):
        gam = self.p["gam"]
        g2 = (gam - 1) / gam
        s = m.al / m.detg
        d = s * u[0]
        ql = [s * (u[4] - u[0]), s * u[1], s * u[2], s * u[3]]
        gss = s * u[5]
        b = [torch.zeros_like(d), s * u[6], s * u[7], s * u[8]]
        bl, qc = self.lower(m, b), self.upper(m, ql)
        bsq = b[1] * bl[1] + b[2] * bl[2] + b[3] * bl[3]
        qb = sum(ql[k] * b[k] for k in range(4))
        qb2 = qb * qb
        z = torch.zeros_like(d)
        on = self.upper(m, [-m.al, z, z, z])
        qn = -qc[0] * m.al
        qt = sum(ql[k] * qc[k] for k in range(4)) + qn * qn
        us = self.qf(m, [None, q[1], q[2], q[3]])
        us = torch.where((us < 0) & (us.abs() <= 1e-4), us.abs(), us)
        us = torch.where(us.abs() > 1e4, torch.full_like(us, 1e4), us)
        gf = torch.sqrt(1 + us)
        vs = us / (1 + us)
        ta, tb, tc = 4 - vs, 4 * (bsq + qn), qt + bsq * bsq + 2 * bsq * qn
        td = torch.sqrt((tb * tb - 4 * ta * tc).abs())
        wp, wm = (-tb + td) / (2 * ta), (-tb - td) / (2 * ta)
        w0 = torch.where(wp > 0, wp, wm)
        none = ~((wp > 0) | (wm >= 0))
        args = (d, gss, bsq, qb, qb2, qn, qt, gf, qc, on, b, m, q, u, at)
        res, wl = self._solve(torch.where(none, torch.ones_like(w0), w0), *args)
        if bool(none.any()):  # W of the cell before it in the loop over k, j, i
            lin = (at[0] * self.shape[1] + at[1]) * self.shape[2] + at[2]
            todo = none.clone()
            for _ in range(64):
                idx = todo.nonzero().flatten()
                if idx.numel() == 0:
                    break
                prev = (idx - 1).clamp(min=0)
                same = (idx > 0) & ((at[1][prev] == at[1][idx]) if self.mink else (idx > 0))
                ready = ~(todo[prev] & same)
                idx, prev, same = idx[ready], prev[ready], same[ready]
                sub = lambda x: x[idx] if isinstance(x, torch.Tensor) else x  # noqa: E731
                ms = _Metric.__new__(_Metric)
                ms.g, ms.c = [[x[idx] for x in r] for r in m.g], [[x[idx] for x in r] for r in m.c]
                ms.detg, ms.al = m.detg[idx], m.al[idx]
                a = [[sub(x) for x in g] if isinstance(g, list) else ms if g is m else sub(g) for g in args[:-1]]
                r2, w2 = self._solve(torch.where(same, wl[prev], torch.zeros_like(wl[prev])), *a, tuple(t[idx] for t in at))
                for v in range(9):
                    res[v][idx] = r2[v]
                wl[idx] = w2
                todo[idx] = False
        return res

    def _solve(self, w, d, gss, bsq, qb, qb2, qn, qt, gf, qc, on, b, m, q, u, at):
        gam = self.p["gam"]
        g1, g2 = gam / (gam - 1), (gam - 1) / gam
        w = w.clone()
        cap = torch.ones_like(w, dtype=torch.bool)
        for _ in range(1000):
            pp = g2 * (w * gf - d * torch.sqrt(gf))
            up = w ** 3 * (w + 2 * bsq) - qb2 * (2 * w + bsq) <= w * w * (qt - bsq * bsq)
            down = ~up & (w ** 3 + w * w * (0.5 * bsq + qn - pp) - 0.5 * qb2 > 0)
            cap = up | down
            if not bool(cap.any()):
                break
            w = torch.where(up, (1.5 * w).abs(), torch.where(down, (float(np.float32(0.9)) * w).abs(), w))
        x = (bsq + w) ** 2
        vs = ((w * w * qt + qb2 * (bsq + 2 * w)) / (w * w * x)).abs()
        vs = torch.where(vs > 1, torch.full_like(vs, 0.99), vs)
        v0 = vs
        W, V = w.clone(), vs.clone()
        live = torch.arange(w.numel(), device=self.dev)[~cap]
        for _ in range(400):  # the two-dimensional iteration; what has not converged by then cycles
            if live.numel() == 0:
                break
            ww, vv, D, B, Q, N, T = W[live], V[live], d[live], bsq[live], qb2[live], qn[live], qt[live]
            gt = 1 - vv
            low = gt < 1e-4
            gt = torch.where(low, torch.full_like(gt, 1e-4), gt)
            vv = torch.where(low, 1 - gt, vv)
            sg = torch.sqrt(gt)
            f = T - vv * (ww + B) ** 2 + Q * (B + 2 * ww) / ww ** 2
            g = -N - 0.5 * B * (1 + vv) + 0.5 * Q / ww ** 2 - ww + g2 * (ww * gt - D * sg)
            fx, fy = -2 * (ww + B) * (vv + Q / ww ** 3), -(ww + B) ** 2
            gx, gy = -1 - Q / ww ** 3 + g2 * gt, -0.5 * B - g2 * ww + 0.5 * g2 * D / sg
            det = fx * gy - fy * gx
            det = torch.where(det == 0, torch.ones_like(det), det)
            dw, dv = (-gy * f + fy * g) / det, (gx * f - fx * g) / det
            ww, vv = torch.clamp((ww + dw).abs(), max=1e5), (vv + dv).abs()
            vv = torch.where(vv > 1, torch.full_like(vv, 0.99), vv)
            W[live], V[live] = ww, vv
            live = live[0.5 * (dw.abs() + dv.abs()) >= 1e-7]
        bad = cap.clone()
        bad[live] = True
        gt = torch.clamp(1 - V, min=1e-4)
        gf = 1 / torch.sqrt(gt)
        ro = d / gf
        pr = g2 * (W * gt - ro)
        second = ((ro < 0) | (pr < 0) | bad) & ~cap
        ut = [None] + [gf / (W + bsq) * (qc[a] + on[a] * qn + qb * b[a] / W) for a in (1, 2, 3)]
        if bool(second.any()):  # the entropy iteration on v^2
            sel = second.nonzero().flatten()
            X, wn = v0[sel].clone(), W[sel].clone()
            D, B, Q, QB, T, G = d[sel], bsq[sel], qb2[sel], qb[sel], qt[sel], gss[sel]
            live = torch.arange(sel.numel(), device=self.dev)
            for _ in range(400):
                if live.numel() == 0:
                    break
                vv = X[live]
                gt = 1 - vv
                low = gt < 1e-4
                gt = torch.where(low, torch.full_like(gt, 1e-4), gt)
                vv = torch.where(low, 1 - gt, vv)
                gg = 1 / torch.sqrt(gt)
                rr = D[live] / gg
                pq = G[live] / D[live] * rr ** gam
                ww = (gg * gg * (rr + g1 * pq)).abs()
                dg = 0.5 * gt ** -1.5
                dw = D[live] * dg + g1 * G[live] * D[live] ** (gam - 1) * (2 - gam) * gg ** (1 - gam) * dg
                f = T[live] - vv * (ww + B[live]) ** 2 + Q[live] * (B[live] + 2 * ww) / ww ** 2
                df = -(ww + B[live]) ** 2 + (-2 * vv * (ww + B[live]) - 2 * Q[live] * (B[live] + 2 * ww) / ww ** 3 + (
                    2 * Q[live] / ww ** 2)) * dw
                step = f / df
                nx = (vv - step).abs()
                X[live] = torch.where(nx >= 1, torch.full_like(nx, 0.99), nx)
                wn[live] = ww
                live = live[step.abs() >= 1e-6]
            gt = torch.clamp(1 - X, min=1e-4)
            gg = 1 / torch.sqrt(gt)
            rr = D / gg
            pq = G / gg * rr ** (gam - 1)
            fde, fpr = self.fde.expand(self.shape)[at][sel], self.fpr.expand(self.shape)[at][sel]
            rr, pq = torch.where(rr < 0, fde, rr), torch.where(pq < 0, fpr, pq)
            ok = torch.ones_like(sel, dtype=torch.bool)
            ok[live] = False
            ww = torch.where(ok, (gg * gg * (rr + g1 * pq)).abs(), wn)
            ro, pr, W, bad = ro.clone(), pr.clone(), W.clone(), bad.clone()
            ro[sel], pr[sel], W[sel], bad[sel] = rr, pq, ww, ~ok
            for a in (1, 2, 3):
                ut[a] = ut[a].clone()
                ut[a][sel] = gg / (ww + B) * (qc[a][sel] + on[a][sel] * qn[sel] + QB * b[a][sel] / ww)
        W = torch.where(cap, w, W)
        new = [ro, ut[1], ut[2], ut[3], pr]
        out = [torch.where(bad, q[v], new[v]) for v in range(5)]
        out.append(torch.where(bad, q[0] * q[4] / q[0] ** gam, ro * pr / ro ** (gam - 1)))
        return out + [u[v] / m.detg for v in (6, 7, 8)], W

    def ghosts(self, q):
        K, J, I = self.shape
        n = self.nm1
        if self.mink:
            for v in range(9):
                q[v][..., :n] = q[v][..., n:n + 1]
                q[v][..., I - n:] = q[v][..., I - n - 1:I - n]
            return
        if not self.jslab:  # phi, over the columns of interior r and theta
            c = (slice(n, K - n), slice(None), slice(n, I - n))
            for v in range(9):
                a = q[v][c]
                a[:, :n] = a[:, J - 2 * n:J - n].clone()
                a[:, J - n:] = a[:, n:2 * n].clone()
        neg = q[1][..., I - n - 1:I - n] < 0
        for v in range(9):
            q[v][..., :n] = q[v][..., n:n + 1]
            last = q[v][..., I - n - 1:I - n]
            q[v][..., I - n:] = torch.where(neg, torch.zeros_like(last), last) if v in (1, 2, 3) else last
        for v in range(9):
            s = -1.0 if v in (3, 8) else 1.0
            q[v][:n] = s * q[v][n:2 * n].flip(0)
            q[v][K - n:] = s * q[v][K - 2 * n:K - n].flip(0)

    def floors(self, q):
        p, m, n = self.p, self.mc, self.nm1
        I = self.shape[2]
        if p["model"] >= 7:
            gf = self.gfl(m, [q[1], q[2], q[3]])
            inflow = (q[1] / gf < 0) & (torch.arange(I, device=self.dev) >= I - n)
            v = [None, (m.be[1] / m.al).expand(self.shape), q[2] / gf, q[3] / gf]
            vs = self.qf(m, v)
            vs = torch.where(vs >= 1, torch.full_like(vs, 0.99), vs)
            g = 1 / torch.sqrt(1 - vs)
            q[1:4] = [torch.where(inflow, v[k] * g, q[k]) for k in (1, 2, 3)]
            thin = (q[0] < 1.01 * self.fde) | ((q[4] < 1.01 * self.fpr) & (q[6] ** 2 + q[7] ** 2 + q[8] ** 2 <= 1e-20))
            q[0], q[4] = torch.where(thin, self.fde, q[0]), torch.where(thin, self.fpr, q[4])
            q[1:4] = [torch.where(thin, torch.zeros_like(q[k]), q[k]) for k in (1, 2, 3)]
            q[5] = torch.zeros_like(q[5])
        de, pr = q[0], q[4]
        gf = self.gfl(m, [q[1], q[2], q[3]])
        v = [None] + [q[k] / gf for k in (1, 2, 3)]
        vs = self.qf(m, v)
        vs = torch.where((vs >= 1) | (gf > 20), torch.full_like(vs, 1 - 1 / 400.0), vs)
        g = 1 / torch.sqrt(1 - vs)
        S = self.state([q[0], v[1] * g, v[2] * g, v[3] * g] + q[4:], m)
        bc = [torch.zeros_like(q[6]), q[6], q[7], q[8]]
        bl = self.lower(m, bc)
        b2 = bc[1] * bl[1] + bc[2] * bl[2] + bc[3] * bl[3]
        f105, f005 = float(np.float32(1.05)), float(np.float32(0.05))
        gg = S["gfl"]
        for _ in range(2000):
            low = (de + p["gam"] / (p["gam"] - 1) * pr) * gg * gg - pr <= (f005 * b2).abs()
            if not bool(low.any()):
                break
            de, pr = torch.where(low, f105 * de, de), torch.where(low, f105 * pr, pr)
        moved = de != q[0]
        r, t = torch.where(moved, de, q[0]), torch.where(~moved & (pr != q[4]), pr, q[4])
        t = torch.where(pr < self.fpr, self.fpr, t)
        t = torch.where(pr > p["pmax"], torch.full_like(t, p["pmax"]), t)
        r = torch.where(de < self.fde, self.fde, r)
        r = torch.where(t / r > 1e6, t / 1e6, r)
        hot, cold = S["bsq"] / r > 50.0, S["bsq"] / t > 2e3
        q[0], q[4] = torch.where(hot, S["bsq"] / 50.0, r), torch.where(cold, S["bsq"] / 2e3, t)

    def step(self, q):
        third, two = float(np.float32(1.0) / np.float32(3.0)), float(np.float32(2.0) / np.float32(3.0))
        dt = self.dt_of(q)
        mask = self.interior()
        un = self.cons(self.state(q, self.mc), self.mc)
        for stage in (1, 2, 3):
            uc = un if stage == 1 else self.cons(self.state(q, self.mc), self.mc)
            F, sf = self.fluxes(q), self.source(q)
            new = []
            for v in range(9):
                L = sum(-(dt / self.dx[d]) * (F[d][v] - self.sh(F[d][v], 3 - d, -1)) for d in (1, 2, 3))
                if 1 <= v <= 4:
                    L = L + dt * sf[v - 1]
                new.append(uc[v] + L if stage == 1 else (3 * un[v] + uc[v]) * 0.25 + 0.25 * L if stage == 2 else
                           (un[v] + 2 * uc[v]) * third + two * L)
            q = self.invert(new, q, mask)
            self.ghosts(q)
            self.floors(q)
        return q

    def load(self, a):
        """Primitives [k, j, i, 9] in the full layout to this run's planes."""
        n = self.nm1
        if self.slab[1] and not self.mink:
            a = a[:, n:n + 1]
        self.shape = tuple(a.shape[:3])
        return [a[..., v].clone() for v in range(9)]


def _advance(p, a, steps):
    """Primitives of one run after `steps` steps, in the full layout."""
    e = _Exact(p)
    q = e.load(a)
    for _ in range(steps):
        q = e.step(q)
    out = torch.stack(q, dim=-1)
    return out.expand(a.shape).contiguous() if e.slab[1] else out


def exact(case, seed):
    grids = _grids(case)
    cells = sum(p["imax"] * p["jmax"] * p["kmax"] for p in grids)
    if case["kind"] != "tubes" and cells > 9_000_000 and case["kind"] == "torus":
        return None  # tens of GB of intermediates
    state = prepare(case, seed)
    if case["kind"] == "calflx":
        p, r = grids[0], state.runs[0]
        e = _Exact(p)
        kk, jj, ii, _ = r.shape
        q = e.load(state.arrays[0].t().reshape(kk, jj, ii, 9).contiguous())
        F = e.fluxes(q)
        return _interior_fluxes(torch.stack([torch.stack(F[d]) for d in (1, 2, 3)]), r)
    inputs = [a.cuda() for a in state.arrays]
    if case["kind"] != "tubes":
        return _by_variable([_advance(p, a, case["steps"]) for p, a in zip(grids, inputs)])
    outs = [None] * len(grids)
    lengths = sorted({p["imax"] for p in grids})
    for n in lengths:  # the tubes of one length side by side
        at = [k for k, p in enumerate(grids) if p["imax"] == n]
        p = grids[at[0]]
        mid = p["jmax"] // 2
        e = _Exact(p)
        stack = torch.cat([inputs[k][mid:mid + 1, mid:mid + 1] for k in at], dim=1)
        e.shape = tuple(stack.shape[:3])
        q = [stack[..., v].clone() for v in range(9)]
        for _ in range(case["steps"]):
            q = e.step(q)
        out = torch.stack(q, dim=-1)
        for c, k in enumerate(at):
            outs[k] = out[:, c:c + 1].expand(inputs[k].shape).contiguous()
    return _by_variable(outs)
