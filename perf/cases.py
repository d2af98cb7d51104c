"""Performance cases: what a user of the solver has it do, through the entry
points of the C ABI (`biocfd.solver.Solver` and `biocfd.adjoint`).

A simulation keeps its blocks registered on the GPU; the library holds one
such registry per process.  A case's blocks, meshes, interfaces and launch
shapes are therefore set up once (`_Session`) and every pass starts from new
fields: it uploads them from pinned host memory (a restart), does its work and
downloads the result (the output files' fields).

Kinds of work:
  run       bcfd_run_steps over all blocks for a few time steps (the native
            driver), mixed precision or FP64, then drag and lift
  dropin    one time step routine by routine, as the Fortran driver calls them
  momentum  nsMomentum2order with the boundary conditions and the forcing
  search    a moved body: normals, tags, lists, normal distances and the
            forcing on the new geometry
  poisson   a zero-boundary Poisson solve and its transpose (the adjoint's)
  adjoint   whole FP64 time steps forward and the discrete adjoint back
"""
import ctypes as C
import json
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "bio-cfd_gb300"))

from biocfd import synth  # noqa: E402
from biocfd._lib import P_d, check  # noqa: E402
from biocfd.adjoint import adjoint_run, poisson_solve, poisson_solve_adjoint  # noqa: E402
from biocfd.solver import Solver  # noqa: E402

DIV_TOL = 1e-6  # residual target of the precisions 1-3 (divergence units)
POISSON_TOL = 1e-10
FIELDS = ("u", "v", "w", "p")


def listed():
    return [
        # two thin plates in tandem at production size (44.0M cells in three
        # blocks), mixed precision with tuned launch shapes: a long run
        {"name": "run_tandem", "kind": "run", "layout": "tandem", "precision": 1, "steps": 2, "tune": True},
        # a coarse and a fine block around a heaving and pitching plate
        # (3.28M cells), mixed precision, from the body's placement on
        {"name": "run_flapping", "kind": "run", "layout": "flapping", "precision": 1, "steps": 4, "tune": True},
        # the two-block sphere (0.66M cells): mixed precision, an ordinary run
        {"name": "run_two_block", "kind": "run", "layout": "pair", "nx": 96, "ny": 64, "nz": 64, "span": 32,
         "body": "sphere", "precision": 1, "steps": 6, "tune": True},
        # a first test of a set-up: one small stretched block of odd sizes,
        # mixed precision, untuned: launches and latency count
        {"name": "run_small", "kind": "run", "layout": "block", "nx": 33, "ny": 21, "nz": 27, "stretch": 1.03,
         "body": "sphere", "precision": 1, "steps": 5, "tune": False},
        # the same driver in FP64 with the reference's arithmetic and stop test
        {"name": "run_fp64", "kind": "run", "layout": "pair", "nx": 96, "ny": 64, "nz": 64, "span": 32,
         "body": "sphere", "precision": 0, "steps": 2, "tune": True},
        # FP64 to a residual target (division-free sweeps), a medium block
        {"name": "run_fp64_target", "kind": "run", "layout": "pair", "nx": 128, "ny": 96, "nz": 96, "span": 64,
         "body": "plate", "precision": 3, "steps": 1, "tune": True},
        # a relinked Fortran driver: the 64^3 sphere routine by routine, FP64
        {"name": "dropin_sphere", "kind": "dropin", "layout": "block", "nx": 64, "ny": 64, "nz": 64, "stretch": 1.0,
         "body": "sphere"},
        # the predictor alone, FP64, on a production fine block with a plate
        {"name": "momentum_large", "kind": "momentum", "layout": "block", "nx": 256, "ny": 192, "nz": 192,
         "stretch": 1.0, "body": "plate"},
        # a moved plate on a medium fine block: re-Search and forcing
        {"name": "search_plate", "kind": "search", "layout": "block", "nx": 160, "ny": 144, "nz": 96, "stretch": 1.0,
         "body": "plate"},
        # pressure solve and its transpose on a stretched block of odd sizes
        {"name": "poisson_pair", "kind": "poisson", "layout": "block", "nx": 97, "ny": 61, "nz": 45, "stretch": 1.02,
         "body": "none"},
        # gradients of drag and lift through two time steps of a sphere
        {"name": "adjoint_sphere", "kind": "adjoint", "layout": "block", "nx": 48, "ny": 48, "nz": 48, "stretch": 1.0,
         "body": "sphere", "steps": 2},
    ]


def _between(rng, lo, hi):
    """An integer spread over the logarithm of [lo, hi]."""
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(("run", "run", "run", "dropin", "momentum", "search", "poisson", "adjoint"))
    c = {"kind": kind, "layout": "block"}
    if kind == "run":
        c["precision"] = rng.choice((1, 1, 1, 0, 2, 3))
        c["steps"] = rng.randint(1, 4)
        c["tune"] = rng.random() < 0.7
        top = 224 if c["precision"] == 1 else 96
        if rng.random() < 0.5:
            n = _between(rng, 24, top)
            c.update(layout="pair", nx=n + rng.randint(0, n // 2), ny=n + rng.randint(0, 5), nz=n - rng.randint(0, 5))
            c["span"] = rng.randint(8, (n - 5) // 2)
            c["body"] = rng.choice(("sphere", "plate"))
            return c
    else:
        top = {"dropin": 80, "momentum": 240, "search": 160, "poisson": 128, "adjoint": 40}[kind]
    n = _between(rng, 20, top)
    c.update(nx=n + rng.randint(0, n // 3), ny=n + rng.randint(-4, 4), nz=n + rng.randint(-4, 4))
    c["stretch"] = rng.choice((1.0, 1.0, 1.01, 1.02))
    c["body"] = {"poisson": "none", "adjoint": "sphere", "search": "plate"}.get(kind) or rng.choice(("sphere", "plate"))
    if kind == "adjoint":
        c["steps"] = rng.randint(1, 2)
    return c


# ---- the simulation's set-up ---------------------------------------------------

def _faces(n, ratio):
    """n cells over [0, n/64], each `ratio` times the one before it up to the middle and back."""
    i = np.arange(n)
    w = ratio ** np.minimum(i, n - 1 - i).astype(np.float64)
    return np.concatenate([[0.0], np.cumsum(w / w.sum())]) * (n / 64.0)


def _block_case(c):
    nx, ny, nz = c["nx"], c["ny"], c["nz"]
    fx, fy, fz = (_faces(n, c["stretch"]) for n in (nx, ny, nz))
    omega = synth.mixed_omega(nx, ny, nz) if c["kind"] == "poisson" or c.get("precision", 0) >= 2 else 1.7
    spec = synth.BlockSpec(nx, ny, nz, fx, fy, fz, omega=omega, is_coarse=True)
    dx = float(min(np.diff(f).min() for f in (fx, fy, fz)))
    mid = np.array([0.45 * fx[-1], 0.5 * fy[-1], 0.5 * fz[-1]])
    size = 0.3 * min(fx[-1], fy[-1], fz[-1])
    if c["body"] == "sphere":
        spec.mesh = synth.fibonacci_sphere(mid, size, dx)
        reach = np.full(3, 0.5 * size)
    elif c["body"] == "plate":
        reach = np.array([size, 0.5 * size, 0.4 * dx])
        spec.mesh = synth.ellipsoid_plate(mid, reach, 0.5 * dx)
    if c["body"] != "none":
        reach = reach + (3.0 * dx if c["kind"] == "search" else 0.0)
        spec.search_box = synth.search_box_for(spec, mid - reach, mid + reach)
    return synth.Case(name="block", blocks=[spec], dt=0.3 * dx, re=200.0 / size, uc=1.0)


def _pair_case(c):
    h = 1.0 / 32.0
    n = np.array([c["nx"], c["ny"], c["nz"]])
    lo = (n - c["span"]) // 2
    box = tuple((float(a * h), float((a + c["span"]) * h)) for a in lo)
    size = 0.4 * c["span"] * h
    case = synth.multi_block(coarse=tuple(int(q) for q in n), domain=tuple(float(q * h) for q in n), fine_boxes=(box,),
                             body=0, diameter=size, reynolds=300.0, plate=c["body"] == "plate",
                             plate_axes=(0.5 * size, 0.25 * size, 0.4 * 0.5 * h))
    return synth.with_mixed_omega(case) if c["precision"] >= 2 else case


def _build(c):
    """The case's blocks; the initial fields come with each state."""
    keep, synth.noisy_initial = synth.noisy_initial, lambda spec, *a, **k: None
    try:
        if c["layout"] == "tandem":
            return synth.tandem_plates()
        if c["layout"] == "flapping":
            return synth.flapping_plate_pair()
        return _pair_case(c) if c["layout"] == "pair" else _block_case(c)
    finally:
        synth.noisy_initial = keep


class _Session:
    """The registered blocks of one case."""

    def __init__(self, c):
        self.case = _build(c)
        self.s = Solver(self.case)
        self.s.setup(with_fields=False)
        if c.get("tune"):
            self.s.autotune()
        if c["kind"] == "poisson":
            # a body-free block is tagged all fluid by the set-up
            check(self.s.L.bcfd_adjoint_set_solver(1), "adjoint_set_solver")

    def bodies(self):
        return [(g, b) for g, b in zip(self.s.handles, self.case.blocks) if b.has_body]

    def place(self, g, b):
        """The body at its start (app/main.F90:64-85): what a new run does first."""
        L, case, m = self.s.L, self.case, b.mesh
        tri = np.ascontiguousarray(m.tris.T, dtype=np.int64)
        xyz = np.ascontiguousarray(m.nodes.T)
        sid = np.ascontiguousarray(m.surf_id, dtype=np.int64)
        check(L.bcfd_block_set_surface(g, len(sid), len(m.nodes), *(_pi(e) for e in tri), _pi(sid),
                                       *(_pd(e) for e in xyz)), "set_surface")
        mo, mi = b.motion, case.motion
        p = np.array([mo.a0_deg, mo.bfreq, mo.yamp, *mo.shift], dtype=np.float64)
        check(L.bcfd_block_set_body_motion(g, _pd(p)), "set_body_motion")
        check(L.bcfd_shift_surface_nodes_initial(g, mi.aoa_deg, mi.piv_pt, 0, case.dt, mi.dxmin, 0.0), "shift_nodes")
        self.tag(g, b)
        self.s.set_time(0, case.dt)

    def tag(self, g, b):
        L = self.s.L
        check(L.bcfd_compute_surface_norm(g, b.mesh.inor), "compute_surface_norm")
        check(L.bcfd_tagging_th(g), "tagging_th")
        check(L.bcfd_cellcount_solid(g), "cellcount_solid")
        check(L.bcfd_compute_norm_distance(g), "compute_norm_distance")
        check(L.bcfd_find_ts_cells(g), "find_ts_cells")


_open = {}  # the one session of this process, by its case


def _session(key):
    if key not in _open:
        _open.clear()
        _open[key] = _Session(json.loads(key))
    return _open[key]


def _pd(a):
    return a.ctypes.data_as(P_d)


def _pi(a):
    return a.ctypes.data_as(C.POINTER(C.c_int64))


def _pt(t):
    return C.cast(t.data_ptr(), P_d)


# ---- inputs ---------------------------------------------------------------------

def _pinned(shape):
    return torch.empty(shape, dtype=torch.float64, pin_memory=True)


def _start_fields(spec, uc, gen):
    """A developed flow's restart: the inflow, a large-scale perturbation and
    fluctuations; arrays are x-fastest, so the tensors' axes are z, y, x."""
    shape = tuple(reversed(spec.shape))
    z, y, x = (torch.linspace(0.0, 2.0 * np.pi, n, device="cuda", dtype=torch.float64) for n in shape)
    out = {}
    for k in FIELDS:
        ph = 6.28 * torch.rand(3, generator=gen, device="cuda", dtype=torch.float64)
        f = torch.sin(z + ph[0])[:, None, None] * torch.sin(y + ph[1])[:, None] * torch.sin(x + ph[2]) * 0.02
        f += torch.randn(shape, generator=gen, device="cuda", dtype=torch.float64) * (1e-3 if k != "p" else 1e-4)
        out[k] = _pinned(shape)
        out[k].copy_(f + uc if k == "u" else f)
    return out


def prepare(case, seed):
    key = json.dumps({k: v for k, v in case.items() if k != "name"}, sort_keys=True)
    sess = _session(key)
    blocks = sess.case.blocks
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    st = {"key": key, "case": dict(case)}
    if case["kind"] == "poisson":
        f = _start_fields(blocks[0], 0.0, gen)
        for name, k in (("r", "v"), ("rt", "w")):
            r = np.zeros(blocks[0].shape, order="F")
            r[1:-1, 1:-1, 1:-1] = f[k].numpy().T[1:-1, 1:-1, 1:-1]
            st[name] = r
        return st
    st["in"] = [_start_fields(b, sess.case.uc, gen) for b in blocks]
    st["out"] = [{k: _pinned(f[k].shape) for k in f} for f in st["in"]]
    if case["kind"] == "search":
        # where the body's motion has taken it: shifted by up to two cells and
        # pitched by up to half a degree about the y axis through its centre
        b = blocks[0]
        st["dist"] = np.zeros(3 * b.nx * b.ny)  # room for any IB list of a plate
        t = (torch.rand(4, generator=gen, device="cuda", dtype=torch.float64) * 2.0 - 1.0).cpu().numpy()
        x, mid = b.mesh.nodes, b.mesh.nodes.mean(axis=0)
        a = t[3] * np.pi / 360.0
        rot = np.array([[np.cos(a), 0.0, np.sin(a)], [0.0, 1.0, 0.0], [-np.sin(a), 0.0, np.cos(a)]])
        st["nodes"] = np.ascontiguousarray(((x - mid) @ rot.T + mid + t[:3] * 2.0 * sess.case.dt / 0.3).T)
    return st


# ---- one pass -------------------------------------------------------------------

def _upload(sess, st):
    for g, f in zip(sess.s.handles, st["in"]):
        u, v, w, p = (_pt(f[k]) for k in FIELDS)
        check(sess.s.L.bcfd_block_upload_fields(g, u, v, w, p, u, v, w), "upload_fields")


def _download(sess, st):
    for g, f in zip(sess.s.handles, st["out"]):
        check(sess.s.L.bcfd_block_download_fields(g, *(_pt(f[k]) for k in FIELDS), None, None, None),
              "download_fields")
    return [f[k] for f in st["out"] for k in FIELDS]


def _ghosts(sess):
    """The thin-surface ghost values of the fields just uploaded."""
    for g, b in sess.bodies():
        check(sess.s.L.bcfd_velocity_forcing_ghost(g), "velocity_forcing_ghost")
        check(sess.s.L.bcfd_pressure_forcing_ghost(g), "pressure_forcing_ghost")


def run(st):
    sess = _session(st["key"])
    s, c = sess.s, st["case"]
    kind = c["kind"]
    if kind == "poisson":
        g = s.handles[0]
        return [poisson_solve(s, g, st["r"], tol=POISSON_TOL), poisson_solve_adjoint(s, g, st["rt"], tol=POISSON_TOL)]
    if kind == "run":
        if sess.case.motion is not None:
            for g, b in sess.bodies():
                sess.place(g, b)
        _upload(sess, st)
        _ghosts(sess)
        s.run(c["steps"], precision=c["precision"], div_tol=DIV_TOL, use_graph=1)
        coef = [s.stress(g, 1.0 / sess.case.re) for g, b in sess.bodies()]
        return _download(sess, st) + coef
    _upload(sess, st)
    if kind == "dropin":
        _ghosts(sess)
        s.step()
        return _download(sess, st)
    if kind == "momentum":
        _ghosts(sess)
        s.momentum_phase()
        # the predictor's results are ut, vt, wt
        o = st["out"][0]
        check(s.L.bcfd_block_download_fields(s.handles[0], None, None, None, None, _pt(o["u"]), _pt(o["v"]), _pt(o["w"])),
              "download_fields")
        return [o["u"], o["v"], o["w"]]
    if kind == "search":
        g, b = sess.bodies()[0]
        check(s.L.bcfd_block_set_nodes(g, *(_pd(e) for e in st["nodes"])), "set_nodes")
        sess.tag(g, b)
        s.research_phase()
        n = s.counts(g)
        dist = s.read(g, "pNormDis", len(st["dist"]))
        st["dist"][:len(dist)], st["dist"][len(dist):] = dist, 0.0
        return _download(sess, st) + [st["dist"], np.array(list(n.values()))]
    # adjoint
    J, duc, grad = adjoint_run(s, {}, c["steps"], every=2, stress_seed=(1.0, 1.0, 1.0, 1.0), mu_f=1.0 / sess.case.re)
    return {"J": J, "duc": duc, **grad}


# ---- the least work, and reference values ------------------------------------------

def work(case):
    """Bytes: every field in and out once per step (FP64) and, for a solve, its
    right-hand side and solution; flops: the predictor's stencil (~450 per
    cell), the correction (~30), per solve and cell one sweep pair's worth of
    updates for each of the n_max pairs an optimally relaxed sweep needs (~14
    per update)."""
    if case["layout"] == "tandem":
        dims = [(384, 256, 256), (256, 192, 192), (256, 192, 192)]
    elif case["layout"] == "flapping":
        dims = [(128, 96, 96), (128, 128, 128)]
    else:
        dims = [(case["nx"], case["ny"], case["nz"])]
        if case["layout"] == "pair":
            dims.append((2 * case["span"],) * 3)
    cells = float(sum(a * b * c for a, b, c in dims))
    pairs = float(sum(a * b * c * max(a, b, c) for a, b, c in dims))
    kind, steps = case["kind"], case.get("steps", 1)
    if kind == "poisson":
        return {"bytes": 2 * 16 * cells, "flops": 2 * 14 * pairs}
    if kind == "momentum":
        return {"bytes": 56 * cells, "flops": 450 * cells}
    if kind == "search":
        return {"bytes": 80 * cells, "flops": 20 * cells}
    step = 14 * pairs + 480 * cells
    if kind == "adjoint":
        return {"bytes": 2 * steps * 64 * cells, "flops": 3 * steps * step}
    return {"bytes": steps * 64 * cells, "flops": steps * step}


def _line(faces, n, sign):
    """The 1-D operator of coefficientMatrix (src/CoefficientMatrix.f90:10-71)
    with its ends folded (sign -1: p = 0 at the face, +1: no gradient)."""
    d = np.diff(faces)
    f = np.concatenate([[faces[0] - d[0]], faces, [faces[-1] + d[-1]]])
    x = 0.5 * (f[1:] + f[:-1])
    a, b = x[1:-1] - x[:-2], x[2:] - x[1:-1]
    lo, di, hi = 2.0 / (a * (a + b)), -2.0 / (a * b), 2.0 / (b * (a + b))
    di[0] += sign * lo[0]
    di[-1] += sign * hi[-1]
    return lo, di, hi


def exact(case, seed):
    """The Poisson solves in closed form: the operator is a sum of three 1-D
    operators, each similar to a symmetric matrix."""
    if case["kind"] != "poisson":
        return None
    st = prepare(case, seed)
    val, q, qi = [], [], []
    for n, sign in ((case["nx"], -1.0), (case["ny"], 1.0), (case["nz"], 1.0)):
        lo, di, hi = _line(_faces(n, case["stretch"]), n, sign)
        s = np.concatenate([[1.0], np.cumprod(np.sqrt(lo[1:] / hi[:-1]))])
        off = np.sqrt(lo[1:] * hi[:-1])
        w, v = np.linalg.eigh(np.diag(di) + np.diag(off, 1) + np.diag(off, -1))
        val.append(w)
        q.append(s[:, None] * v)
        qi.append(v.T / s[None, :])
    lam = val[0][:, None, None] + val[1][None, :, None] + val[2][None, None, :]

    def solve(r, p, pi):
        t = np.einsum("ai,bj,ck,ijk->abc", *pi, r, optimize=True) / lam
        x = np.zeros(tuple(n + 2 for n in t.shape), order="F")
        x[1:-1, 1:-1, 1:-1] = np.einsum("ai,bj,ck,ijk->abc", *p, t, optimize=True)
        return x

    inner = (slice(1, -1),) * 3
    return [solve(st["r"][inner], q, qi), solve(st["rt"][inner], [m.T for m in qi], [m.T for m in q])]
