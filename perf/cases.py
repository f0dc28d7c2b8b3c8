"""What a user of the solver has it do, as cases that can be timed.

Each case is one call (or one burst of requests) through the public API:

  solve     one frequency in FP64, what the reference's main program does:
            GHMATECD + LINSOLVE + un-swap (BemSolver.solve_frequency)
  sweep     a frequency sweep of one mesh (BemSolver.sweep), mixed or plain
  batch     many small meshes of uneven size in one call (batch_solve)
  static    the static diagonals every new mesh needs (BemSolver.ghmatece)
  assemble  GHMATECD into a device buffer of the caller (bem_ghmatecd_noalloc)
  interior  displacements and stresses at interior points (BemSolver.interior)
  serve     a burst of requests with new boundary values for problems the
            server holds (right-hand-side-only solves)

Meshes are the repository's own kind: a jittered nx x ny grid of boundary
elements over [-5, 5]^2, closed by non-collocated enclosing elements, with
NPG = 4 (the synthetic workloads), 6 or 8 (the reference's shipped cases).
Loads are a unit traction patch; `clamped` elements (|x| beyond a limit) have
prescribed displacements (KODE = 0), which takes the column swap.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from __graft_entry__ import load_package

load_package()
from bem_mececcs_b200 import capi, meshgen, serve  # noqa: E402
from bem_mececcs_b200.solver import BemSolver, batch_solve  # noqa: E402


# ---------------------------------------------------------------------------
# The cases.
# ---------------------------------------------------------------------------

def listed() -> list:
    return [
        # The smallest everyday call: one frequency of the 240-element mesh,
        # where launches and the latency of each pivot column count.
        dict(name="solve_240", kind="solve", nx=16, ny=15, npg=4, nu=0.25, damping=0.01, clamped=0.0),
        # The reference's own soil-trench size and rule (510 elements, NPG = 8,
        # nu = 0.3, no damping), here with a clamped strip.
        dict(name="solve_510_npg8_clamped", kind="solve", nx=30, ny=17, npg=8, nu=0.3, damping=0.0,
             clamped=3.5),
        # The headline mesh solved one frequency at a time in FP64.
        dict(name="solve_2160", kind="solve", nx=48, ny=45, npg=4, nu=0.25, damping=0.01, clamped=0.0),
        # A sweep of a small mesh: many lockstep problems of 720 unknowns.
        dict(name="sweep_240_mixed", kind="sweep", nx=16, ny=15, npg=4, nu=0.25, damping=0.01, clamped=0.0,
             count=32, form="mixed", refine=3),
        # A medium mesh of odd size, an odd number of frequencies, clamped
        # elements: nothing is a multiple of a tile.
        dict(name="sweep_957_mixed_clamped", kind="sweep", nx=33, ny=29, npg=4, nu=0.3, damping=0.02,
             clamped=3.5, count=13, form="mixed", refine=3),
        # The same class of work in the plain FP64 form.
        dict(name="sweep_600_plain", kind="sweep", nx=25, ny=24, npg=4, nu=0.25, damping=0.01, clamped=0.0,
             count=9, form="plain", refine=0),
        # The headline: the 2160-element sweep in the mixed form with the
        # benchmark's two refinement steps (28 of its 128 frequencies).
        dict(name="sweep_2160_mixed", kind="sweep", nx=48, ny=45, npg=4, nu=0.25, damping=0.01, clamped=0.0,
             count=28, form="mixed", refine=2),
        # The largest mesh of the precision form, one frequency (n = 25920).
        dict(name="sweep_8640_mixed", kind="sweep", nx=96, ny=90, npg=4, nu=0.25, damping=0.01, clamped=0.0,
             count=1, form="mixed", refine=3),
        # Many users' small meshes at once, n = 75..1800, each its own material.
        dict(name="batch_96_mixed", kind="batch", count=96, lo=24, hi=600, form="mixed", refine=3),
        # The static diagonals of the headline mesh: paid for every new mesh.
        dict(name="static_2160", kind="static", nx=48, ny=45, npg=4, nu=0.25),
        # The assembly alone at the reference's rule, 1600 elements, NPG = 8.
        dict(name="assemble_1600_npg8", kind="assemble", nx=40, ny=40, npg=8, nu=0.3, damping=0.0,
             clamped=0.0),
        # Interior results: the reference evaluates points below a solved surface.
        dict(name="interior_960_pts1000", kind="interior", nx=32, ny=30, npg=4, nu=0.25, damping=0.01,
             points=1000, stresses=True),
    ]


def _grid(rng, lo, hi):
    """nx x ny with lo <= nx*ny <= hi elements, sizes spread over the logarithm."""
    while True:
        e = math.exp(rng.uniform(math.log(lo), math.log(hi)))
        ny = max(2, int(round(math.sqrt(e / rng.uniform(1.0, 1.6)))))
        nx = max(ny, int(round(e / ny)))
        if lo <= nx * ny <= hi:
            return nx, ny


def draw(rng) -> dict:
    kind = rng.choice(["solve", "solve", "sweep", "sweep", "sweep", "batch", "static", "assemble", "interior",
                       "serve"])
    mat = dict(nu=round(rng.uniform(0.15, 0.35), 3), damping=round(rng.choice([0.0, rng.uniform(0.005, 0.05)]), 4))
    clamped = rng.choice([0.0, 0.0, round(rng.uniform(2.5, 4.0), 2)])
    if kind == "solve":
        npg = rng.choice([4, 4, 6, 8])
        nx, ny = _grid(rng, 90, 2160 if npg == 4 else 1200)
        return dict(kind=kind, nx=nx, ny=ny, npg=npg, clamped=clamped, **mat)
    if kind == "sweep":
        form = rng.choice(["mixed", "mixed", "mixed", "plain"])
        npg = rng.choice([4, 4, 4, 8])
        nx, ny = _grid(rng, 90, (2160 if npg == 4 else 1200) if form == "mixed" else 900)
        count = rng.randint(1, 28 if nx * ny > 500 else 64) if form == "mixed" else rng.randint(1, 12)
        return dict(kind=kind, nx=nx, ny=ny, npg=npg, clamped=clamped, count=count, form=form,
                    refine=rng.choice([2, 3]) if form == "mixed" else 0, **mat)
    if kind == "batch":
        lo = rng.randint(20, 60)
        return dict(kind=kind, count=rng.randint(5, 96), lo=lo, hi=rng.randint(2 * lo, 600),
                    form=rng.choice(["mixed", "mixed", "plain"]), refine=3)
    if kind == "static":
        nx, ny = _grid(rng, 90, 4000)
        return dict(kind=kind, nx=nx, ny=ny, npg=rng.choice([4, 6, 8]) if nx * ny < 2000 else 4, nu=mat["nu"])
    if kind == "assemble":
        npg = rng.choice([4, 6, 8])
        nx, ny = _grid(rng, 90, {4: 3000, 6: 2000, 8: 1600}[npg])
        return dict(kind=kind, nx=nx, ny=ny, npg=npg, clamped=clamped, **mat)
    if kind == "interior":
        nx, ny = _grid(rng, 90, 2160)
        return dict(kind=kind, nx=nx, ny=ny, npg=rng.choice([4, 8]) if nx * ny < 1000 else 4,
                    points=int(math.exp(rng.uniform(math.log(10), math.log(1500)))),
                    stresses=rng.random() < 0.7, **mat)
    # requests for problems the server holds: a new right-hand side each
    nx, ny = _grid(rng, 240, 1200)
    return dict(kind="serve", nx=nx, ny=ny, count=rng.randint(1, 8), refine=rng.choice([2, 3]), **mat)


# ---------------------------------------------------------------------------
# Inputs, from the seed alone.
# ---------------------------------------------------------------------------

def _rng(seed, *more):
    return np.random.Generator(np.random.PCG64([int(seed), *more]))


def _mesh(case, rng):
    return meshgen.enclosed_grid(case["nx"], case["ny"], jitter=0.10, seed=int(rng.integers(1 << 30)),
                                 npg=case["npg"], rnu=case["nu"], depth=2.5, layers=4)


def _load(mesh, rng, damping, clamped, spacing):
    """A unit traction patch somewhere on the surface; the elements beyond
    |x| = clamped have zero displacement prescribed."""
    d = meshgen.traction_patch(mesh, radius=max(1.0, 1.3 * spacing), dam=damping,
                               center=(float(rng.uniform(-2, 2)), float(rng.uniform(-3, 3))))
    if clamped:
        cxm = mesh.centroids()[0][: mesh.nbe]
        held = np.repeat(np.abs(cxm) > clamped, 3)
        d.kode[held] = 0
        d.bc[held] = 0.0
    return d


def _omegas(rng, count):
    """Log-uniform in [0.1, 10], the sweep's range."""
    return np.exp(rng.uniform(np.log(0.1), np.log(10.0), size=count))


def _inputs(case, seed):
    """Everything the case works on, on the host."""
    rng = _rng(seed)
    kind = case["kind"]
    if kind == "batch":
        # the sizes belong to the case; jitter, materials and loads to the seed
        sizes = _rng(case["count"], case["lo"], case["hi"])
        probs = []
        for _ in range(case["count"]):
            nx, ny = serve.grid_for(int(sizes.integers(case["lo"], case["hi"] + 1)))
            one = dict(nx=nx, ny=ny, npg=4, nu=float(rng.uniform(0.15, 0.35)))
            m = _mesh(one, rng)
            d = _load(m, rng, float(rng.uniform(0.005, 0.05)), 0.0, 10.0 / ny)
            probs.append((m, d, float(rng.uniform(0.1, 10.0))))
        return dict(probs=probs)
    spacing = 10.0 / min(case["nx"], case["ny"])
    if kind == "serve":
        m = _mesh(dict(case, npg=4), rng)
        fr = _omegas(rng, case["count"])
        loads = [[_load(m, rng, case["damping"], 0.0, spacing).bc.astype(np.complex128) for _ in range(2)]
                 for _ in range(case["count"])]
        return dict(mesh=m, freqs=fr, loads=loads, kode=np.ones(3 * m.nbe, dtype=np.int32),
                    material=(m.ge, m.rnu, case["damping"], 1.0))
    m = _mesh(case, rng)
    out = dict(mesh=m)
    if kind == "static":
        return out
    d = out["load"] = _load(m, rng, case["damping"], case.get("clamped", 0.0), spacing)
    out["freqs"] = _omegas(rng, case.get("count", 1))
    if kind == "interior":
        # boundary values as a solved surface has them: smooth, decaying from
        # the load, displacements everywhere and tractions under the patch
        cxm, cym, _ = m.centroids()
        x, y = cxm[: m.nbe], cym[: m.nbe]
        k = float(out["freqs"][0])
        amp = rng.standard_normal(3) + 1j * rng.standard_normal(3)
        r = np.sqrt(1.0 + x * x + y * y)
        out["disp"] = ((np.exp(-1j * k * r) / r)[:, None] * amp[None, :]).ravel()
        out["trac"] = d.bc.astype(np.complex128)
        pts = case["points"]
        out["points"] = (rng.uniform(-4.5, 4.5, pts), rng.uniform(-4.5, 4.5, pts), rng.uniform(-2.0, -0.5, pts))
    return out


def _solver(mesh, load=None):
    """A mesh on the GPU with its static diagonals and boundary values."""
    sol = BemSolver(mesh, device=0)
    if load is not None:
        sol.ghmatece()
        sol.set_bc(load.kode, load.bc.astype(np.complex128), load.dam, load.rho)
    return sol


def prepare(case, seed):
    kind = case["kind"]
    x = _inputs(case, seed)
    st = dict(case=case, kind=kind)
    if kind == "batch":
        st["problems"] = [(_solver(m, d), fr) for m, d, fr in x["probs"]]
        st["driver"] = capi.Context(0)
        return st
    if kind == "serve":
        srv = serve.Server(budget_bytes=60e9, form="mixed", refine=case["refine"])
        mid = srv.add_mesh(x["mesh"])
        # the problems' first solves: the server keeps their factors
        first = [srv.submit(mid, x["material"], fr, bc[0], x["kode"]) for fr, bc in zip(x["freqs"], x["loads"])]
        for r in first:
            srv.wait(r)
        st.update(server=srv, mesh_id=mid, material=x["material"], kode=x["kode"],
                  requests=[(float(fr), bc[1]) for fr, bc in zip(x["freqs"], x["loads"])])
        return st
    st["solver"] = sol = _solver(x["mesh"], x.get("load"))
    if "freqs" in x:
        st["freqs"] = x["freqs"]
    if kind == "sweep":
        st["batch"] = min(case["count"], sol.sweep_batch_limit(case["form"]))
    elif kind == "assemble":
        # column-major nn x (nn + 1): torch's rows are the system's columns
        st["a"] = torch.empty(sol.nn + 1, sol.nn, dtype=torch.complex128, device="cuda")
    elif kind == "interior":
        st.update(disp=x["disp"], trac=x["trac"], points=x["points"])
    return st


# ---------------------------------------------------------------------------
# One pass.
# ---------------------------------------------------------------------------

def run(state):
    case, kind = state["case"], state["kind"]
    if kind == "batch":
        xs, _ = batch_solve(state["driver"], state["problems"], form=case["form"], refine=case["refine"])
        return np.concatenate(xs)
    if kind == "serve":
        srv = state["server"]
        ids = [srv.submit(state["mesh_id"], state["material"], fr, bc, state["kode"])
               for fr, bc in state["requests"]]
        return np.stack([srv.wait(i)[0] for i in ids])
    sol = state["solver"]
    if kind == "solve":
        disp, trac = sol.solve_frequency(float(state["freqs"][0]))
        return dict(disp=disp, trac=trac)
    if kind == "sweep":
        # the second result is each problem's last correction: a measure of
        # convergence at rounding level, not a computed quantity
        return sol.sweep(state["freqs"], form=case["form"], batch=state["batch"], refine=case["refine"])[0]
    if kind == "static":
        hd, gd = sol.ghmatece()
        return dict(hestdiag=hd, gestdiag=gd)
    if kind == "interior":
        zd, zs = sol.interior(float(state["freqs"][0]), state["disp"], state["trac"], *state["points"],
                              stresses=case["stresses"])
        return dict(zdsol=zd) if zs is None else dict(zdsol=zd, zssol=zs)
    zge, zcs, zcp = (capi.f64([z.real, z.imag]) for z in sol.material)
    a = state["a"]
    sol.ctx.check(sol.ctx.L.bem_ghmatecd_noalloc(
        sol.ctx.h, capi.ptr(zge), capi.ptr(zcs), capi.ptr(zcp), capi.ptr(capi.f64(sol.c)),
        float(state["freqs"][0]), capi.BEM_FAST_SINGULAR, a.data_ptr(), sol.nn), "bem_ghmatecd_noalloc")
    return a


# ---------------------------------------------------------------------------
# What a pass cannot do without.
# ---------------------------------------------------------------------------

# Real operations of one Stokes evaluation (complex U and T at one Gauss point
# and their weighted sums), of one Kelvin T and of one interior stress
# evaluation.
_STOKES, _KELVIN, _STRESS = 613.0, 110.0, 1500.0


def _enclosed_count(case):
    nx, ny = case["nx"], case["ny"]
    return 2 * nx * ny + 4 * 2 * (nx + ny)


def _lu(n):
    return 8.0 / 3.0 * n ** 3 + 8.0 * n * n


def work(case) -> dict:
    kind = case["kind"]
    if kind == "batch":
        mid = [case["lo"] + (case["hi"] - case["lo"]) * (i + 0.5) / case["count"] for i in range(case["count"])]
        return dict(bytes=sum(3 * e * 16 * 2 for e in mid),
                    flops=sum(_lu(3 * e) + _STOKES * e * e * 16 for e in mid))
    nbe = case["nx"] * case["ny"]
    n = 3 * nbe
    if kind == "serve":  # G times the new values, one solve and `refine` corrections, per request
        steps = case["refine"]
        per = 8.0 * n * n * (2 + 2 * steps)
        return dict(bytes=case["count"] * (16.0 * n * n * 2 + 8.0 * n * n), flops=case["count"] * per)
    ng = case["npg"] ** 2
    if kind == "static":
        return dict(bytes=_enclosed_count(case) * 150.0 + 144.0 * nbe, flops=_KELVIN * nbe * _enclosed_count(case) * ng)
    if kind == "interior":
        per = _STOKES + (_STRESS if case["stresses"] else 0.0)
        return dict(bytes=nbe * 250.0 + case["points"] * 220.0, flops=per * nbe * case["points"] * ng)
    assembly = _STOKES * nbe * nbe * ng
    if kind == "assemble":
        return dict(bytes=16.0 * n * (n + 1), flops=assembly)
    count = case.get("count", 1)
    return dict(bytes=count * 32.0 * n, flops=count * (assembly + _lu(n)))


# ---------------------------------------------------------------------------
# The same results in 64 bits, in plain torch.
# ---------------------------------------------------------------------------

def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _t(a):
    return torch.as_tensor(np.ascontiguousarray(a), device=_dev())


class _Geometry:
    """Gauss points, weights, normals and centroids of all elements."""

    def __init__(self, m):
        node = np.stack([m.cx, m.cy, m.cz], 1)
        self.co = co = node[np.asarray(m.cone) - 1]                      # [N, 4, 3]
        self.n, self.nbe = m.n, m.nbe
        self.rule = np.polynomial.legendre.leggauss(m.npg)
        nrm = np.cross(co[:, 1] - co[:, 0], co[:, 2] - co[:, 0])
        self.normal = _t(nrm / np.linalg.norm(nrm, axis=1, keepdims=True))
        self.centre = _t(co.mean(1))
        p, w = self.points(co)
        self.p, self.w = _t(p), _t(w)                                    # [ng, N, 3], [ng, N]

    def points(self, co):
        gi, om = self.rule
        g1, g2 = (a.ravel() for a in np.meshgrid(gi, gi, indexing="ij"))
        wt = np.outer(om, om).ravel()
        shape = 0.25 * np.stack([(1 - g1) * (1 - g2), (1 + g1) * (1 - g2), (1 + g1) * (1 + g2), (1 - g1) * (1 + g2)])
        d1 = 0.25 * np.stack([-(1 - g2), 1 - g2, 1 + g2, -(1 + g2)])
        d2 = 0.25 * np.stack([-(1 - g1), -(1 + g1), 1 + g1, 1 - g1])
        det = np.linalg.norm(np.cross(np.einsum("kg,nkc->gnc", d1, co), np.einsum("kg,nkc->gnc", d2, co)), axis=2)
        return np.einsum("kg,nkc->gnc", shape, co), wt[:, None] * det


def _rel(points, x):
    """r, r/|r| of points [N, 3] seen from x [R, 3]."""
    d = [points[None, :, c] - x[:, None, c] for c in range(3)]
    r = torch.sqrt(d[0] ** 2 + d[1] ** 2 + d[2] ** 2)
    return r, [v / r for v in d]


def _dot3(a, b):
    return a[0] * b[0] + a[1] * b[1] + a[2] * b[2]


def _kelvin_t(c, r, rd, nv, i, j):
    drn = _dot3(rd, nv)
    dl = 1.0 if i == j else 0.0
    return c[2] / r ** 2 * (drn * (c[3] * dl + 3 * rd[i] * rd[j]) + c[3] * (rd[j] * nv[i] - rd[i] * nv[j]))


def _static_consts(m):
    return (1 / (16 * math.pi * m.ge * (1 - m.rnu)), 3 - 4 * m.rnu, -1 / (8 * math.pi * (1 - m.rnu)), 1 - 2 * m.rnu)


def _exact_static(m, g):
    """HESTdiag by the rigid-body row sums and GESTdiag by four collapsed
    triangles, both [nbe, 3 (j), 3 (i)]."""
    c = _static_consts(m)
    hd = torch.zeros(g.nbe, 3, 3, dtype=torch.float64, device=_dev())
    nv = [g.normal[None, :, k] for k in range(3)]
    step = max(1, 8_000_000 // g.n)
    for lo in range(0, g.nbe, step):
        rows = torch.arange(lo, min(g.nbe, lo + step), device=_dev())
        for q in range(g.p.shape[0]):
            r, rd = _rel(g.p[q], g.centre[rows])
            w = g.w[q][None, :].expand_as(r).clone()
            w[torch.arange(len(rows), device=_dev()), rows] = 0.0       # the element itself
            for j in range(3):
                for i in range(3):
                    hd[rows, j, i] -= (w * _kelvin_t(c, r, rd, nv, i, j)).sum(1)
    gd = torch.zeros_like(hd)
    mid = g.co[: g.nbe].mean(1)
    for k in range(4):
        co = np.stack([g.co[: g.nbe, k], g.co[: g.nbe, (k + 1) % 4], mid, mid], 1)
        p, w = (_t(a) for a in g.points(co))
        d = p - g.centre[None, : g.nbe]
        r = d.norm(dim=2)
        rd = d / r[..., None]
        for j in range(3):
            for i in range(3):
                gd[:, j, i] += (w * c[0] / r * (c[1] * (i == j) + rd[..., i] * rd[..., j])).sum(0)
    return hd, gd


class _Medium:
    """The complex material and the radial functions of the dynamic kernels."""

    def __init__(self, m, damping, fr, rho=1.0):
        self.zge = complex(m.ge, 2 * m.ge * damping)
        self.zcs = complex(np.sqrt(np.complex128(self.zge / rho)))
        self.zcp = self.zcs * math.sqrt((2 - 2 * m.rnu) / (1 - 2 * m.rnu))
        self.kp, self.ks = -1j * fr / self.zcp, -1j * fr / self.zcs
        self.q, self.rho = (self.zcs / self.zcp) ** 2, rho
        self.c0 = 1 / (4 * math.pi * self.zge)

    def radial(self, r):
        p, s = self.kp * r, self.ks * r
        ep, es = torch.exp(p), torch.exp(s)
        q = self.q
        f = (1 + 1 / s ** 2 - 1 / s) * es / r - q * (1 / p ** 2 - 1 / p) * ep / r
        k = (1 + 3 / s ** 2 - 3 / s) * es / r - q * (1 + 3 / p ** 2 - 3 / p) * ep / r
        fr = (-2 + s + 3 / s - 3 / s ** 2) * es / r ** 2 - q * (-1 + 3 / p - 3 / p ** 2) * ep / r ** 2
        kr = (s - 4 + 9 / s - 9 / s ** 2) * es / r ** 2 - q * (p - 4 + 9 / p - 9 / p ** 2) * ep / r ** 2
        aa = fr - k / r
        bb = 4 * k / r - 2 * kr
        cc = (1 / q - 2) * (aa + bb / 2 - 3 * k / r) - 2 * k / r
        return f, k, fr, kr, aa, bb, cc

    def second(self, r):
        """Second derivatives for the stresses."""
        a, b = -self.kp * r, -self.ks * r
        ea, eb = torch.exp(-a), torch.exp(-b)
        f2 = (-(self.q * ea * (12 + 12 * a + 5 * a ** 2 + a ** 3) / (a ** 2 * r ** 3)) +
              eb * (12 + 12 * b + 7 * b ** 2 + 3 * b ** 3 + b ** 4) / (b ** 2 * r ** 3))
        k2 = (-(self.q * ea * (36 + 36 * a + 17 * a ** 2 + 5 * a ** 3 + a ** 4) / (a ** 2 * r ** 3)) +
              eb * (36 + 36 * b + 17 * b ** 2 + 5 * b ** 3 + b ** 4) / (b ** 2 * r ** 3))
        return f2, k2


def _exact_system(m, g, hd, gd, medium, kode, zdfi):
    """The swapped H [nn, nn] and the right-hand side."""
    c = _static_consts(m)
    nbe, nn = g.nbe, 3 * g.nbe
    H = torch.empty(nn, nn, dtype=torch.complex128, device=_dev())
    rhs = torch.empty(nn, dtype=torch.complex128, device=_dev())
    nv = [g.normal[None, :nbe, k] for k in range(3)]
    held = _t(np.asarray(kode) == 0)
    zdfi = _t(np.asarray(zdfi, dtype=np.complex128))
    step = max(1, 3_000_000 // nbe)
    for lo in range(0, nbe, step):
        rows = torch.arange(lo, min(nbe, lo + step), device=_dev())
        at = torch.arange(len(rows), device=_dev())
        h = torch.zeros(len(rows), 3, nbe, 3, dtype=torch.complex128, device=_dev())
        u = torch.zeros_like(h)
        for q in range(g.p.shape[0]):
            r, rd = _rel(g.p[q, :nbe], g.centre[rows])
            f, k, _, _, aa, bb, cc = medium.radial(r)
            w = g.w[q, None, :nbe]
            drn = _dot3(rd, nv)
            r0, rd0 = r[at, rows], [v[at, rows] for v in rd]
            n0, w0 = [v[0, rows] for v in nv], w[0, rows]
            for i in range(3):
                for j in range(3):
                    dl = 1.0 if i == j else 0.0
                    u[:, i, :, j] += w * medium.c0 * (f * dl - k * (rd[i] * rd[j]))
                    h[:, i, :, j] += w / (4 * math.pi) * (aa * (drn * dl + rd[j] * nv[i]) + bb * (rd[i] * rd[j] * drn) +
                                                         cc * (rd[i] * nv[j]))
                    # the element itself: the static kernels are taken out here
                    # and added below as the static diagonals
                    u[at, i, rows, j] -= w0 * c[0] / r0 * (c[1] * dl + rd0[i] * rd0[j])
                    h[at, i, rows, j] -= w0 * _kelvin_t(c, r0, rd0, n0, i, j)
        h[at, :, rows, :] += hd[rows].transpose(1, 2)
        u[at, :, rows, :] += gd[rows].transpose(1, 2)
        h, u = h.reshape(3 * len(rows), nn), u.reshape(3 * len(rows), nn)
        h, u = torch.where(held, -u, h), torch.where(held, -h * medium.zge, u)
        H[3 * lo:3 * lo + h.shape[0]] = h
        rhs[3 * lo:3 * lo + h.shape[0]] = u @ zdfi
        del h, u
    return H, rhs


def _exact_solution(m, load_bc, kode, damping, freqs, many_loads=False):
    g = _Geometry(m)
    hd, gd = _exact_static(m, g)
    out = []
    for i, fr in enumerate(freqs):
        bc = load_bc[i] if many_loads else load_bc
        H, rhs = _exact_system(m, g, hd, gd, _Medium(m, damping, float(fr)), kode, bc)
        out.append(torch.linalg.solve(H, rhs).cpu().numpy())
        del H, rhs
    return np.stack(out)


def _exact_interior(m, x, case):
    g = _Geometry(m)
    md = _Medium(m, case["damping"], float(x["freqs"][0]))
    pts = _t(np.stack(x["points"], 1))
    nbe, L = g.nbe, len(pts)
    u = [_t(x["disp"].reshape(nbe, 3)[:, k])[None, :] for k in range(3)]
    t = [_t(x["trac"].reshape(nbe, 3)[:, k])[None, :] for k in range(3)]
    nv = [g.normal[None, :nbe, k] for k in range(3)]
    nu = _dot3(u, nv)
    zd = torch.zeros(L, 3, dtype=torch.complex128, device=_dev())
    zs = torch.zeros(L, 3, 3, dtype=torch.complex128, device=_dev())    # [point, j, i]
    mu, lm = md.zge, (md.zcp ** 2 * md.rho - 2 * md.zge) / md.zge
    for q in range(g.p.shape[0]):
        r, rd = _rel(g.p[q, :nbe], pts)
        f, k, fr, kr, aa, bb, cc = md.radial(r)
        w = g.w[q, None, :nbe]
        drn, rt, ru = _dot3(rd, nv), _dot3(rd, t), _dot3(rd, u)
        for i in range(3):
            uu = md.c0 * (f * t[i] - k * (rd[i] * rt))
            tt = (aa * (drn * u[i] + nv[i] * ru) + bb * (rd[i] * drn * ru) + cc * (rd[i] * nu)) / (4 * math.pi)
            zd[:, i] += (w * (uu - tt)).sum(1)
        if not case["stresses"]:
            continue
        f2, k2 = md.second(r)
        c1 = 2 * k / r
        c2 = lm * (fr - kr - c1)
        c3 = fr - k / r
        c4 = 2 * (kr - c1)
        c5 = 4 * (k2 - 5 * kr / r + 8 * k / r ** 2)
        c6 = f2 - fr / r - 3 * kr / r + 6 * k / r ** 2
        c9 = 2 * (2 * kr / r - 4 * k / r ** 2 + lm * (k2 + kr / r - 4 * k / r ** 2 - f2 + fr / r))
        c10 = 4 * k / r ** 2 + 4 * lm * (kr / r + 2 * k / r ** 2 - fr / r)
        c11 = lm ** 2 * (k2 + 4 * kr / r + 2 * k / r ** 2 - f2 - 2 * fr / r)
        c12 = 2 * (fr / r - k / r ** 2)
        for i in range(3):
            for j in range(3):
                dl = 1.0 if i == j else 0.0
                d = (c1 - c2) * dl * rt - c3 * (rd[i] * t[j] + t[i] * rd[j]) + c4 * (rd[i] * rd[j]) * rt
                s = (drn * (c5 * (rd[i] * rd[j]) * ru - c6 * (u[j] * rd[i] + u[i] * rd[j]) + c9 * dl * ru) +
                     c9 * (rd[i] * rd[j]) * nu - c6 * (rd[i] * nv[j] + rd[j] * nv[i]) * ru + (c10 + c11) * dl * nu -
                     c12 * (u[i] * nv[j] + u[j] * nv[i]))
                zs[:, j, i] += (w * (d - mu * s)).sum(1) / (4 * math.pi)
    out = dict(zdsol=zd.reshape(-1).cpu().numpy())
    if case["stresses"]:
        out["zssol"] = zs.reshape(-1).cpu().numpy()
    return out


def exact(case, seed):
    kind = case["kind"]
    x = _inputs(case, seed)
    if kind == "batch":
        return np.concatenate([_exact_solution(m, d.bc, d.kode, d.dam, [fr])[0] for m, d, fr in x["probs"]])
    m = x["mesh"]
    if kind == "serve":
        return _exact_solution(m, [bc[1] for bc in x["loads"]], x["kode"], case["damping"], x["freqs"], many_loads=True)
    if kind == "interior":
        return _exact_interior(m, x, case)
    if kind == "static":
        hd, gd = _exact_static(m, _Geometry(m))
        return dict(hestdiag=hd.cpu().numpy().ravel(), gestdiag=gd.cpu().numpy().ravel())
    d = x["load"]
    if kind == "assemble":
        g = _Geometry(m)
        hd, gd = _exact_static(m, g)
        H, rhs = _exact_system(m, g, hd, gd, _Medium(m, case["damping"], float(x["freqs"][0])), d.kode, d.bc)
        return torch.cat([H.T, rhs[None, :]])
    sol = _exact_solution(m, d.bc, d.kode, case["damping"], x["freqs"])
    if kind == "sweep":
        return sol
    held = d.kode == 0
    zge = complex(m.ge, 2 * m.ge * case["damping"])
    return dict(disp=np.where(held, d.bc, sol[0]).astype(np.complex128),
                trac=np.where(held, sol[0] * zge, d.bc).astype(np.complex128))
