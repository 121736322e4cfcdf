"""The pressure-solve work a flow solver gives this library, as measurable cases.

Every case is one call (or the few calls of one time step) through the public
Python entry points, on the default device layout: whole solves on uniform and
adaptive meshes in the three precisions, from host arrays and from device
tensors; the merged batch of independent problems; the differentiable solve,
forward and backward; the two-phase time step (coefficients, hierarchy refresh,
force, projection); its field kernels alone; and the two-block capillary-wave
solve.  Sizes are those of `tpagmg.workloads`, of the tests and of `bench.py`,
and generic ones around them: blocks of 6 to 16 cells, periodic and walled
sides, domains from 1,024 to 4.2 million cells, trees of 1 to 6 levels.

`exact` restates the equations in FP64 with numpy and torch alone (FFT on the
uniform meshes, the face-metric operator and plain conjugate gradients on the
trees); of the library it takes only the mesh's index arrays, which are inputs.
"""
import functools
import math
import os
import pathlib
import sys
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import torch

sys.path.insert(0, str(pathlib.Path(__file__).resolve().parents[1] / "twophaseamr.jl_b200"))

import tpagmg  # noqa: E402
from tpagmg import projection as P  # noqa: E402
from tpagmg import workloads as W  # noqa: E402
from tpagmg.adjoint import pressure_solve  # noqa: E402
from tpagmg.cmdgfm import solve_cmdgfm  # noqa: E402
from tpagmg.operator import mixture_density  # noqa: E402

RTOL = 1e-10            # the reference's `solve!` default
CENTER = (0.5, 0.6)     # the droplet of `workloads.droplet_spec`
SIGMA = 0.072


# ---- the cases ---------------------------------------------------------------

def listed():
    return [
        # the smallest pressure solve: four blocks in a closed box, called on
        # host arrays as a Julia `ccall` would (launches and latency)
        dict(name="box_32_host_mixed", kind="uniform", nx=32, ny=32, bx=16, by=16, px=False, py=False,
             precision="mixed", host=True),
        # the single-phase projection of a Taylor-Green flow, in FP64
        dict(name="periodic_128_fp64", kind="uniform", nx=128, ny=128, bx=16, by=16, px=True, py=True,
             precision="fp64", host=False),
        # an odd channel: blocks of 10 x 6, periodic along, walls across, host arrays
        dict(name="channel_240x144_fp64", kind="uniform", nx=240, ny=144, bx=10, by=6, px=True, py=False,
             precision="fp64", host=True),
        # a periodic 2:1 domain with FP32 Krylov vectors in FP64 refinement
        dict(name="periodic_1024x512_ir", kind="uniform", nx=1024, ny=512, bx=16, by=16, px=True, py=True,
             precision="mixed_ir", host=False),
        # the large uniform solve (4.2 million cells)
        dict(name="periodic_2048_mixed", kind="uniform", nx=2048, ny=2048, bx=16, by=16, px=True, py=True,
             precision="mixed", host=False),
        # a two-phase droplet on a shallow tree, plain FP64
        dict(name="droplet_l3_fp64", kind="droplet", levels=3, radius=0.15, ratio=1000.0, precision="fp64"),
        # the headline solve: the two-phase droplet, 110k cells, mixed precision
        dict(name="droplet_l4_mixed", kind="droplet", levels=4, radius=0.15, ratio=1000.0, precision="mixed"),
        # gradients with respect to the right-hand side and 1/rho: forward and backward
        dict(name="droplet_l2_gradient", kind="gradient", levels=2, radius=0.15, ratio=1000.0, precision="fp64"),
        # one two-phase time step's pressure part, all fields on the device
        dict(name="droplet_l4_step", kind="step", levels=4, radius=0.15, ratio=1000.0, precision="mixed"),
        # the step's field kernels on a deep tree
        dict(name="droplet_l6_fields", kind="fields", levels=6, radius=0.15, ratio=1000.0),
        # independent problems of uneven depth, solved together
        dict(name="batch_16_mixed", kind="batch", count=16, draw_seed=W.SEEDS["batch"], precision="mixed"),
        # the capillary wave's two-velocity system (nonsymmetric, jump block)
        dict(name="wave_l6_two_block", kind="wave", levels=6, precision="mixed"),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["uniform", "uniform", "uniform", "droplet", "droplet", "gradient", "step", "fields", "batch",
                       "wave"])
    precision = rng.choice(["fp64", "mixed", "mixed_ir"])
    if kind == "uniform":
        bx, by = rng.choice([(16, 16), (16, 16), (16, 16), (8, 8), (10, 6), (12, 16)])
        # block counts (1..3) x 2^k: the tree coarsens while both counts are even
        ox, oy = rng.choice([(1, 1), (1, 1), (1, 2), (2, 1), (1, 3), (3, 1)] + [(3, 3)] * (bx * by < 100))
        k = max(1, round(0.5 * math.log2(_log(rng, 1024, 2.0e6) / (ox * bx * oy * by))))
        nx, ny = ox * bx << k, oy * by << k
        return dict(kind=kind, nx=nx, ny=ny, bx=bx, by=by, px=rng.random() < 0.6, py=rng.random() < 0.6,
                    precision=precision, host=rng.random() < 0.3)
    radius, ratio = round(rng.uniform(0.08, 0.28), 3), rng.choice([10.0, 100.0, 1000.0])
    if kind == "droplet":
        return dict(kind=kind, levels=rng.randint(1, 5), radius=radius, ratio=ratio, precision=precision)
    if kind == "gradient":
        return dict(kind=kind, levels=rng.randint(1, 4), radius=radius, ratio=ratio,
                    precision=rng.choice(["fp64", "mixed"]))
    if kind == "step":
        return dict(kind=kind, levels=rng.randint(2, 4), radius=radius, ratio=ratio,
                    precision=rng.choice(["fp64", "mixed"]))
    if kind == "fields":
        return dict(kind=kind, levels=rng.randint(2, 6), radius=radius, ratio=ratio)
    if kind == "batch":
        return dict(kind=kind, count=rng.randint(2, 16), draw_seed=rng.randrange(1, 10000),
                    precision=rng.choice(["fp64", "mixed"]))
    return dict(kind=kind, levels=rng.randint(2, 6), precision=rng.choice(["fp64", "mixed"]))


# ---- meshes, coefficients and right-hand sides ----------------------------------

def _uniform_mesh(c):
    return tpagmg.BlockTreeMesh(base_mesh=(c["nx"], c["ny"]), block_size=(c["bx"], c["by"]),
                                extent=(c["nx"] / c["ny"], 1.0), periodic=(c["px"], c["py"]))


@functools.lru_cache(maxsize=3)
def _uniform_solver(nx, ny, bx, by, px, py):
    """A uniform domain's solver, made once: a program keeps it for all its
    right-hand sides (the set-up of 4.2 million cells takes 11 s on the host)."""
    mesh = _uniform_mesh(dict(nx=nx, ny=ny, bx=bx, by=by, px=px, py=py))
    return tpagmg.EllipticSolver(tpagmg.PoissonOperator(mesh, 1.0))


def _lattice_rhs(c, seed):
    """Zero-mean N(0, 1) noise per cell of the nx x ny lattice (row-major in y)."""
    f = W.rng(seed).standard_normal((c["ny"], c["nx"]))
    return f - f.mean()


def _to_cells(c, field):
    """Lattice field -> the mesh's cell order (row-major blocks, cells row-major inside)."""
    by, bx = c["by"], c["bx"]
    return np.ascontiguousarray(field.reshape(c["ny"] // by, by, c["nx"] // bx, bx).transpose(0, 2, 1, 3).ravel())


def _droplet(c, seed):
    """Mesh, fractions and 1/rho of a droplet; the centre moves with the seed
    by at most two finest cells, well inside the refined band."""
    g = W.rng(seed)
    h = 1.0 / (64 << c["levels"])
    center = (CENTER[0] + h * g.uniform(-2, 2), CENTER[1] + h * g.uniform(-2, 2))
    mesh = tpagmg.BlockTreeMesh(**W.droplet_spec(levels=c["levels"], radius=c["radius"], center=CENTER))
    frac = W.circle_fractions(mesh, center, c["radius"])
    kappa = 1.0 / mixture_density(mesh, frac, (c["ratio"], 1.0))
    return mesh, frac, kappa


def _potential(c, frac):
    return SIGMA / c["radius"] * (frac > 0.5).astype(np.float64)


def _velocity(mesh, seed):
    """A predicted face velocity: a smooth vortex and 1 % noise."""
    x, y = mesh.face_centers()
    u = np.where(mesh.face_axis == 1, np.sin(np.pi * x) * np.cos(np.pi * y), -np.cos(np.pi * x) * np.sin(np.pi * y))
    return u + 0.01 * W.rng(seed + 1).standard_normal(mesh.nfaces)


def _batch(c):
    problems = W.batch_problems(c["count"], c["draw_seed"])
    with ThreadPoolExecutor(min(16, os.cpu_count() or 1)) as ex:
        meshes = list(ex.map(lambda p: tpagmg.BlockTreeMesh(**W.batch_spec(p)), problems))
        inputs = list(ex.map(lambda mp: W.batch_inputs(*mp), zip(meshes, problems)))
    return problems, meshes, [k for k, _ in inputs]


def _batch_rhs(meshes, seed):
    return [W.gaussian_rhs(m, 1000 * seed + k) for k, m in enumerate(meshes)]


def _gradient_target(mesh, seed):
    return 1e-3 * W.rng(seed + 2).standard_normal(mesh.ncells)


def _wave(c, seed):
    mesh = tpagmg.BlockTreeMesh(**W.capillary_wave_spec(c["levels"]))
    frac = W.wave_fractions(mesh)
    kappa = 1.0 / mixture_density(mesh, frac, (1.0, 1e-3))
    solver = tpagmg.EllipticSolver(tpagmg.PoissonOperator(mesh, kappa))
    system, truth = W.cmdgfm_system(mesh, solver.level_matrix(0), kappa, frac, seed=seed)
    return solver, system, truth


def _cuda(a):
    return torch.from_numpy(np.ascontiguousarray(a, dtype=np.float64)).cuda()


# ---- a program's state and one pass ------------------------------------------------

def prepare(case, seed):
    c, kind = case, case["kind"]
    if kind == "uniform":
        solver = _uniform_solver(c["nx"], c["ny"], c["bx"], c["by"], c["px"], c["py"])
        rhs = _to_cells(c, _lattice_rhs(c, seed))
        if c["host"]:
            return dict(case=c, solver=solver, rhs=rhs, x=np.zeros_like(rhs))
        rhs = _cuda(rhs)
        return dict(case=c, solver=solver, rhs=rhs, x=torch.zeros_like(rhs))
    if kind == "droplet":
        mesh, frac, kappa = _droplet(c, seed)
        solver = tpagmg.EllipticSolver(tpagmg.PoissonOperator(mesh, kappa))
        rhs = _cuda(W.droplet_rhs(mesh, solver.apply(_potential(c, frac)), seed))
        return dict(case=c, solver=solver, rhs=rhs, x=torch.zeros_like(rhs))
    if kind == "gradient":
        mesh, frac, kappa = _droplet(c, seed)
        solver = tpagmg.EllipticSolver(tpagmg.PoissonOperator(mesh, kappa))
        return dict(case=c, solver=solver, rhs=_cuda(W.gaussian_rhs(mesh, seed)).requires_grad_(),
                    kappa=_cuda(kappa).requires_grad_(), target=_cuda(_gradient_target(mesh, seed)))
    if kind == "step":
        mesh, frac, kappa = _droplet(c, seed)
        solver = tpagmg.EllipticSolver(tpagmg.PoissonOperator(mesh, kappa),
                                       preconditioner_options={"precision": c["precision"]})
        step = P.TwoPhaseStep(solver, (c["ratio"], 1.0), sigma=SIGMA, curvature=1.0 / c["radius"])
        return dict(case=c, solver=solver, step=step, fraction=_cuda(frac), velocity=_cuda(_velocity(mesh, seed)),
                    boundary=torch.zeros(mesh.nboundary_faces, dtype=torch.float64, device="cuda"),
                    pressure=torch.zeros(mesh.ncells, dtype=torch.float64, device="cuda"))
    if kind == "fields":
        mesh, frac, kappa = _droplet(c, seed)
        solver = tpagmg.EllipticSolver(tpagmg.PoissonOperator(mesh, kappa))
        out = {k: torch.zeros(n, dtype=torch.float64, device="cuda") for k, n in
               dict(physical=mesh.ncells, conditional=mesh.ncells, kappa=mesh.nfaces, force=mesh.nfaces,
                    gradient=mesh.nfaces, divergence=mesh.ncells).items()}
        return dict(case=c, solver=solver, fraction=_cuda(frac), velocity=_cuda(_velocity(mesh, seed)),
                    boundary=torch.zeros(mesh.nboundary_faces, dtype=torch.float64, device="cuda"),
                    pressure=_cuda(W.rng(seed + 3).standard_normal(mesh.ncells)), out=out)
    if kind == "batch":
        problems, meshes, kappas = _batch(c)
        with ThreadPoolExecutor(min(16, os.cpu_count() or 1)) as ex:
            solvers = list(ex.map(lambda mk: tpagmg.EllipticSolver(tpagmg.PoissonOperator(*mk)), zip(meshes, kappas)))
        batch = tpagmg.BatchedSolver(solvers)
        rhs = _cuda(batch.concat(_batch_rhs(meshes, seed)))
        return dict(case=c, solver=batch, rhs=rhs, x=torch.zeros_like(rhs))
    solver, system, _ = _wave(c, seed)
    return dict(case=c, solver=solver, system=system)


def _stream():
    return torch.cuda.current_stream().cuda_stream


def run(state):
    c, s = state["case"], state["solver"]
    kind = c["kind"]
    if kind == "uniform" and c["host"]:
        x = state["x"]
        x[:] = 0.0
        tpagmg.solve(x, s, state["rhs"], rtol=RTOL, precision=c["precision"])
        return {"pressure": x}
    if kind in ("uniform", "droplet", "batch"):
        x = state["x"]
        x.zero_()
        s.set_stream(_stream())
        s.solve_device(state["rhs"].data_ptr(), x.data_ptr(), rtol=RTOL, precision=c["precision"])
        return {"pressure": x}
    if kind == "gradient":
        p = pressure_solve(state["rhs"], state["kappa"], s, rtol=1e-11, precision=c["precision"])
        loss = 0.5 * ((p - state["target"]) ** 2).sum()
        rhs_bar, kappa_bar = torch.autograd.grad(loss, (state["rhs"], state["kappa"]))
        return {"pressure": p.detach(), "rhs_bar": rhs_bar, "kappa_bar": kappa_bar}
    if kind == "step":
        step, dt = state["step"], 1e-3
        step.update_interface(state["fraction"])
        u = state["velocity"] + dt * step.force()
        ub, p = state["boundary"].clone(), state["pressure"].clone()
        step.project(u, ub, p, dt, tolerance=1e-11)
        return {"velocity": u, "pressure": p, "kappa": step.kappa}
    if kind == "fields":
        o, density = state["out"], (c["ratio"], 1.0)
        P.conditional_fraction_device(s, state["fraction"], o["conditional"], o["physical"])
        P.face_coefficients_device(s, o["conditional"], density, o["kappa"])
        P.surface_tension_device(s, o["conditional"], o["force"], sigma=SIGMA, curvature=1.0 / c["radius"])
        P.weighted_gradient_device(s, state["pressure"], o["gradient"])
        P.divergence_device(s, state["velocity"], state["boundary"], o["divergence"])
        return dict(o)
    x, _ = solve_cmdgfm(s, state["system"], precision=c["precision"])
    return {"solution": x}


# ---- compulsory work ------------------------------------------------------------------

@functools.lru_cache(maxsize=64)
def _tree_sizes(levels, radius):
    m = tpagmg.BlockTreeMesh(**W.droplet_spec(levels=levels, radius=radius, center=CENTER))
    return m.ncells, m.nfaces


def work(case):
    """Inputs read once and outputs written once; operations of one operator
    product (a solve needs many, but how many is the method's choice)."""
    c, kind = case, case["kind"]
    if kind == "uniform":
        n = c["nx"] * c["ny"]
        return {"bytes": 16 * n, "flops": 10 * n}
    if kind == "batch":
        meshes = [tpagmg.BlockTreeMesh(**W.batch_spec(p)) for p in W.batch_problems(c["count"], c["draw_seed"])]
        n, nf = sum(m.ncells for m in meshes), sum(m.nfaces for m in meshes)
        return {"bytes": 16 * n + 8 * nf, "flops": 10 * n}
    if kind == "wave":
        m = tpagmg.BlockTreeMesh(**W.capillary_wave_spec(c["levels"]))
        return {"bytes": 16 * m.ncells + 60 * m.ncells, "flops": 10 * m.ncells}  # vectors and the CSR matrix
    n, nf = _tree_sizes(c["levels"], c["radius"])
    if kind == "droplet":
        return {"bytes": 16 * n + 8 * nf, "flops": 10 * n}
    if kind == "gradient":  # rhs, target, p, rhs_bar; kappa, kappa_bar
        return {"bytes": 32 * n + 16 * nf, "flops": 20 * n + 8 * nf}
    if kind == "step":      # fraction, two pressures; velocity in and out, kappa
        return {"bytes": 24 * n + 24 * nf, "flops": 10 * n + 20 * nf}
    # fields: fraction, pressure, physical, conditional, divergence; velocity, kappa, force, gradient
    return {"bytes": 40 * n + 32 * nf, "flops": 10 * n + 20 * nf}


# ---- 64-bit values ----------------------------------------------------------------------

def _fft_solution(c, seed):
    """-div grad p = f on the uniform lattice: FFT along periodic axes, even
    reflection (a cosine transform) along walled ones."""
    f = torch.from_numpy(_lattice_rhs(c, seed))
    f = f.cuda() if torch.cuda.is_available() else f
    ny, nx = f.shape
    hx, hy = c["nx"] / c["ny"] / nx, 1.0 / ny
    if not c["px"]:
        f = torch.cat([f, f.flip(1)], 1)
    if not c["py"]:
        f = torch.cat([f, f.flip(0)], 0)
    my, mx = f.shape
    kx = torch.arange(mx // 2 + 1, device=f.device, dtype=torch.float64)
    ky = torch.arange(my, device=f.device, dtype=torch.float64)
    lam = (2 / hy * torch.sin(math.pi * ky / my))[:, None] ** 2 + (2 / hx * torch.sin(math.pi * kx / mx))[None] ** 2
    lam[0, 0] = 1.0
    p = torch.fft.rfft2(f) / lam
    p[0, 0] = 0.0
    return torch.fft.irfft2(p, s=(my, mx))[:ny, :nx].cpu().numpy()


def _face_metric(m):
    """The inverse face metric K (faces x faces) as a torch sparse CSR matrix.

    Per lattice vertex with the faces that end there: 1 / (2 |f| d_f) on the
    diagonal beside walls and where at most two faces meet; elsewhere
    N (M'N)^-1 N' + (tr / (n - 2)) (1 - M (M'M)^-1 M'), with rows |f| (dx, dy)
    of M and half unit normals in N."""
    nxb, nyb = m.block_size
    lev = m.keys[:, 0].max()
    lat = np.array([m.base_mesh[0] << lev, m.base_mesh[1] << lev], dtype=np.int64)

    def bounds(cells):
        b, r = cells // (nxb * nyb), cells % (nxb * nyb)
        s = 1 << (lev - m.keys[b, 0]).astype(np.int64)
        return np.stack([(m.keys[b, 1] * np.int64(nxb) + r % nxb) * s, (m.keys[b, 2] * np.int64(nyb) + r // nxb) * s]), s

    (lo_m, s_m), (lo_p, s_p) = bounds(m.face_minus), bounds(m.face_plus)
    nf, a = m.nfaces, m.face_axis.astype(np.int64) - 1
    t, f = 1 - a, np.arange(m.nfaces)
    per = np.array(m.periodic)
    normal = lo_m[a, f] + s_m
    normal = np.where(per[a], normal % lat[a], normal)
    ends = np.stack([np.maximum(lo_m[t, f], lo_p[t, f]), np.minimum(lo_m[t, f] + s_m, lo_p[t, f] + s_p)])
    bm, bp = m.face_minus // (nxb * nyb), m.face_plus // (nxb * nyb)
    dn = (m.spacing[bm, a] + m.spacing[bp, a]) / 2
    off = 2 * lo_p[t, f] + s_p - 2 * lo_m[t, f] - s_m
    off = np.where(per[t] & (off > lat[t]), off - 2 * lat[t], off)
    off = np.where(per[t] & (off < -lat[t]), off + 2 * lat[t], off)
    dt = off * (np.array(m.extent)[t] / lat[t] / 2)
    d = np.where(a == 0, [dn, dt], [dt, dn])
    vx = np.where(a == 0, normal, ends)
    vy = np.where(a == 0, ends, normal)
    vx, vy = (np.where(per[k], v % lat[k], v) for k, v in ((0, vx), (1, vy)))
    key, who = (vx * (lat[1] + 1) + vy).ravel(), np.tile(f, 2)
    order = np.argsort(key, kind="stable")
    key, who = key[order], who[order]
    first = np.nonzero(np.r_[True, key[1:] != key[:-1]])[0]
    count = np.diff(np.r_[first, len(key)])
    kx, ky = key[first] // (lat[1] + 1), key[first] % (lat[1] + 1)
    wall = (not per[0]) & ((kx == 0) | (kx == lat[0])) | (not per[1]) & ((ky == 0) | (ky == lat[1]))
    plain = wall | (count <= 2)
    rows, cols, vals = [], [], []
    for n in np.unique(count):
        at = first[(count == n) & plain]
        if len(at):
            w = (at[:, None] + np.arange(n)).ravel()
            rows.append(who[w])
            cols.append(who[w])
            vals.append(0.5 / (m.face_area[who[w]] * dn[who[w]]))
        at = first[(count == n) & ~plain]
        if len(at):
            w = who[at[:, None] + np.arange(n)]
            M = m.face_area[w][..., None] * np.moveaxis(d[:, w], 0, -1)
            N = 0.5 * (a[w][..., None] == np.arange(2))
            mn = np.swapaxes(M, 1, 2) @ N
            cons = N @ np.linalg.solve((mn + np.swapaxes(mn, 1, 2)) / 2, np.swapaxes(N, 1, 2))
            proj = np.eye(n) - M @ np.linalg.solve(np.swapaxes(M, 1, 2) @ M, np.swapaxes(M, 1, 2))
            loc = cons + np.trace(cons, axis1=1, axis2=2)[:, None, None] / (n - 2) * proj
            rows.append(np.repeat(w, n, axis=1).ravel())
            cols.append(np.tile(w, (1, n)).ravel())
            vals.append(((loc + np.swapaxes(loc, 1, 2)) / 2).ravel())
    return _sparse(np.concatenate(rows), np.concatenate(cols), np.concatenate(vals), (nf, nf))


def _sparse(rows, cols, vals, shape):
    t = torch.sparse_coo_tensor(torch.from_numpy(np.stack([rows, cols])), torch.from_numpy(vals), shape)
    t = t.coalesce().to_sparse_csr()
    return t.cuda() if torch.cuda.is_available() else t


class _Tree:
    """S = J' sqrt(k) K sqrt(k) J of a closed tree mesh, J the area-weighted jump."""

    def __init__(self, mesh, kappa):
        f = np.arange(mesh.nfaces)
        rows, cols = np.r_[f, f], np.r_[mesh.face_minus, mesh.face_plus]
        vals = np.r_[-mesh.face_area, mesh.face_area]
        self.J, self.Jt = (_sparse(rows, cols, vals, (mesh.nfaces, mesh.ncells)),
                           _sparse(cols, rows, vals, (mesh.ncells, mesh.nfaces)))
        self.K = _face_metric(mesh)
        self.dev = self.K.device
        self.v = self.t(mesh.cell_volumes())
        self.area2 = self.t(mesh.face_area ** 2)
        self.cells = [torch.from_numpy(c.astype(np.int64)).to(self.dev) for c in (mesh.face_minus, mesh.face_plus)]
        crow, col, val = self.K.crow_indices(), self.K.col_indices(), self.K.values()
        row = torch.repeat_interleave(torch.arange(mesh.nfaces, device=self.dev), crow[1:] - crow[:-1])
        self.Kd = torch.zeros(mesh.nfaces, dtype=torch.float64, device=self.dev).index_add_(
            0, row[row == col], val[row == col])
        self.coefficients(kappa)

    def coefficients(self, kappa):
        self.sk = self.t(np.sqrt(kappa))
        fd = self.Kd * self.sk ** 2 * self.area2
        self.diag = torch.zeros_like(self.v)  # of K's diagonal: the preconditioner below
        for c in self.cells:
            self.diag.index_add_(0, c, fd)

    def t(self, a):
        return torch.from_numpy(np.ascontiguousarray(a, dtype=np.float64)).to(self.dev)

    def gradient(self, p):
        return self.sk * (self.K @ (self.sk * (self.J @ p)))

    def apply(self, p):
        return self.Jt @ self.gradient(p)

    def solve(self, strong):
        """G S^+ Pi (V f): zero volume mean; CG with the diagonal, restarted on true residuals."""
        b = self.v * strong
        b = b - self.v * (b.sum() / self.v.sum())
        x = torch.zeros_like(b)
        scale = float((b / self.v).abs().max())
        for _ in range(6):
            r = b - self.apply(x)
            r = r - self.v * (r.sum() / self.v.sum())
            stop = max(1e-9 * float((r / self.v).abs().max()), 1e-14 * scale)
            if float((r / self.v).abs().max()) <= 1e-13 * scale:
                break
            e, z = torch.zeros_like(b), r / self.diag
            q, rz = z.clone(), torch.dot(r, z)
            for it in range(60000):
                s = self.apply(q)
                alpha = rz / torch.dot(q, s)
                e.add_(alpha * q)
                r.sub_(alpha * s)
                z = r / self.diag
                new = torch.dot(r, z)
                q.mul_(new / rz).add_(z)
                rz = new
                if it % 100 == 99 and float((r / self.v).abs().max()) <= stop:
                    break
            x += e
        return x - (self.v * x).sum() / self.v.sum()

    def kappa_gradient(self, p, lam):
        """-lam' (dS/dkappa_f) p per face."""
        u, w = self.J @ p, self.J @ lam
        return -0.5 * (w * (self.K @ (self.sk * u)) + u * (self.K @ (self.sk * w))) / self.sk


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind == "uniform":
        return {"pressure": _to_cells(c, _fft_solution(c, seed))}
    if kind == "wave":  # the right-hand side is the product of this vector
        return {"solution": _wave(c, seed)[2]}
    if kind == "batch":
        if c["count"] > 4:
            return None  # plain conjugate gradients on every problem: more than 20 s
        problems, meshes, kappas = _batch(c)
        if sum(m.ncells for m in meshes) > 300_000:
            return None
        return {"pressure": np.concatenate([T.solve(T.t(r)).cpu().numpy() for T, r in
                                            zip(map(_Tree, meshes, kappas), _batch_rhs(meshes, seed))])}
    mesh, frac, kappa = _droplet(c, seed)
    if kind != "fields" and mesh.ncells > 250_000:
        return None  # tens of thousands of plain iterations
    tree = _Tree(mesh, kappa)
    if kind == "droplet":
        rhs = W.droplet_rhs(mesh, tree.apply(tree.t(_potential(c, frac))).cpu().numpy(), seed)
        return {"pressure": tree.solve(tree.t(rhs)).cpu().numpy()}
    if kind == "gradient":
        p = tree.solve(tree.t(W.gaussian_rhs(mesh, seed)))
        lam = tree.solve((p - tree.t(_gradient_target(mesh, seed))) / tree.v)
        return {"pressure": p.cpu().numpy(), "rhs_bar": (tree.v * lam).cpu().numpy(),
                "kappa_bar": tree.kappa_gradient(p, lam).cpu().numpy()}
    # the fraction floor of the two-phase fields is sqrt(eps): below it a cell counts as empty, above 1 - it as full
    floor = math.sqrt(np.finfo(np.float64).eps)
    cond = np.where(frac <= floor, 0.0, np.where(frac >= 1 - floor, 1.0, frac))
    kappa_c = 1.0 / mixture_density(mesh, cond, (c["ratio"], 1.0))
    jump = SIGMA / c["radius"] * ((cond[mesh.face_plus] > 0.5) * 1.0 - (cond[mesh.face_minus] > 0.5)) * mesh.face_area
    u = _velocity(mesh, seed)

    def divergence(v):
        return -(tree.Jt @ tree.t(v)) / tree.v

    if kind == "fields":
        force = tree.sk * (tree.K @ (tree.sk * tree.t(jump)))
        return {"physical": cond, "conditional": cond, "kappa": kappa_c, "force": force.cpu().numpy(),
                "gradient": tree.gradient(tree.t(W.rng(seed + 3).standard_normal(mesh.ncells))).cpu().numpy(),
                "divergence": divergence(u).cpu().numpy()}
    dt = 1e-3
    tree.coefficients(kappa_c)
    u = tree.t(u) + dt * (tree.sk * (tree.K @ (tree.sk * tree.t(jump))))
    phi = tree.solve((tree.Jt @ u) / tree.v / dt)
    return {"velocity": (u - dt * tree.gradient(phi)).cpu().numpy(), "pressure": phi.cpu().numpy(), "kappa": kappa_c}
