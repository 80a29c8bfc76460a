"""Workloads of the leap-frog engine as its users run it, for timing.

A case is a dict of plain values. Five kinds of use:

  run     a prepared simulation advances `steps` leap-frog steps and hands
          back what it recorded: every receiver sample of every shot and the
          final wavefield of every shot (Simulation.run / seismograms /
          u_all). One shot is forward modelling; several shots on one mesh
          are a survey. `op` is the stored operator or the matrix-free one.
  batch   independent meshes of uneven size and degree advanced together
          (Batch), each with its own material, time step and source.
  cfl     the power iteration behind the time step (Simulation.estimate_lmax).
  survey  the whole program for one model of an inversion or a parameter
          sweep: create the simulation from mesh and material arrays, set the
          sources, run, read the shot gathers, release it.

Meshes are jittered rectangles (two triangles per square), vp is log-normal
per element (sigma 0.1, vs = vp / sqrt 3, rho 2300), sources are Ricker forces
and receivers lie a fraction of an element below the top surface, all drawn
from the seed. Results of FP32-operator simulations are kept in float32, the
precision such gathers are stored in; FP64 results stay float64.

exact() is the same recurrence with the assembled interior-penalty operator
in plain torch float64, from its own mesh, basis and quadrature code.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from tspeed_b200 import capi
from tspeed_b200.workloads import Mesh, Problem, Source

PENALTY = 10.0
VP, RHO = 3000.0, 2300.0
WEIGHT = {"fp64": 8, "fp32": 4, "bf16": 2}


# ------------------------------------------------------------------ cases --
def listed():
    return [
        # A homogeneous-size tutorial model: 1,600 triangles, one shot. The
        # operator fits in L2; a step lasts microseconds.
        dict(name="run1_n4_small", kind="run", N=4, nx=40, ny=20, shots=1, nrcv=8, precision="fp64", op="explicit",
             steps=2000),
        # The plain drop-in: 40,000 triangles, degree 5, FP64 blocks, one shot.
        dict(name="run1_n5_fp64", kind="run", N=5, nx=200, ny=100, shots=1, nrcv=128, precision="fp64",
             op="explicit", steps=400),
        # One large shot with FP32 blocks: 160,000 triangles, degree 6 (8 GB of operator).
        dict(name="run1_n6_fp32", kind="run", N=6, nx=400, ny=200, shots=1, nrcv=64, precision="fp32", op="explicit",
             steps=300),
        # The same mesh without stored blocks, the form for meshes whose operator is too large to keep.
        dict(name="run1_n6_matfree", kind="run", N=6, nx=400, ny=200, shots=1, nrcv=64, precision="fp64",
             op="matrix_free", steps=400),
        # A small odd-sized mesh at low degree, matrix-free.
        dict(name="run1_n3_matfree", kind="run", N=3, nx=91, ny=37, shots=1, nrcv=21, precision="fp64",
             op="matrix_free", steps=1000),
        # A 64-shot survey, FP32 operator (10,000 triangles, degree 5).
        dict(name="run64_n5_fp32", kind="run", N=5, nx=100, ny=50, shots=64, nrcv=128, precision="fp32",
             op="explicit", steps=1000),
        # The same survey in exact FP64.
        dict(name="run64_n5_fp64", kind="run", N=5, nx=100, ny=50, shots=64, nrcv=128, precision="fp64",
             op="explicit", steps=600),
        # A survey whose shot count fills no tile: 24 shots, degree 4.
        dict(name="run24_n4_fp32", kind="run", N=4, nx=121, ny=60, shots=24, nrcv=48, precision="fp32", op="explicit",
             steps=1000),
        # A handful of shots at high degree, FP64.
        dict(name="run6_n7_fp64", kind="run", N=7, nx=70, ny=35, shots=6, nrcv=32, precision="fp64", op="explicit",
             steps=500),
        # Sixteen meshes of 500 to 20,000 triangles, degrees 3 to 8, FP32 blocks.
        dict(name="batch16_fp32", kind="batch", meshes=16, tri_min=500, tri_max=20000, n_min=3, n_max=8, nrcv=8,
             precision="fp32", op="explicit", steps=100),
        # Time-step selection on the drop-in's mesh.
        dict(name="cfl_n5", kind="cfl", N=5, nx=200, ny=100, shots=1, nrcv=8, precision="fp64", op="explicit",
             steps=100),
        # One model of a sweep end to end: 8 shots, 500 steps.
        dict(name="survey8_n4_fp64", kind="survey", N=4, nx=80, ny=40, shots=8, nrcv=64, precision="fp64",
             op="explicit", steps=500),
    ]


def draw(rng):
    def logint(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    kind = rng.choice(["run", "run", "run", "run", "matfree", "matfree", "batch", "cfl", "survey"])
    nrcv = logint(4, 128)
    if kind == "batch":
        lo = rng.randint(3, 5)
        return dict(kind="batch", meshes=rng.randint(2, 20), tri_min=500, tri_max=logint(1000, 12000), n_min=lo,
                    n_max=rng.randint(lo, 8), nrcv=rng.randint(1, 12), precision=rng.choice(["fp32", "fp64"]),
                    op="explicit", steps=rng.randint(40, 80))
    N = rng.randint(3, 8)
    if kind == "matfree":
        ne = logint(1600, 120000)
        shots, prec, op = 1, "fp64", "matrix_free"
    elif kind == "run":
        shots = rng.choice([1, 1, logint(2, 64), logint(2, 96)])
        prec, op = rng.choice(["fp64", "fp32"]), "explicit"
        ne = logint(800, 40000) if shots == 1 else logint(800, 12000)
    else:
        shots = 1 if kind == "cfl" else logint(1, 32)
        prec, op = rng.choice(["fp64", "fp32"]), "explicit"
        ne = logint(800, 20000)
    ny = max(4, int(round(math.sqrt(ne / 2 / rng.uniform(1.0, 3.0)))))
    nx = max(4, ne // 2 // ny)
    # Long runs on small models, bounded work on large ones.
    cost = 2 * nx * ny * (N + 1) ** 4 * max(1.0, shots / 8.0)
    steps = int(min(1500, max(60, 6e9 / cost)))
    if kind == "cfl":
        steps = min(steps, 150)
    return dict(kind="run" if kind == "matfree" else kind, N=N, nx=nx, ny=ny, shots=shots, nrcv=nrcv, precision=prec,
                op=op, steps=steps)


# ----------------------------------------------------------------- models --
def _mesh(nx, ny, h, rng):
    """Vertices and triangles of an nx x ny grid of squares of side h, each
    split along its rising diagonal, interior vertices moved by up to 10 % of
    h; triangles counter-clockwise, two per square, row by row."""
    i, j = np.meshgrid(np.arange(nx + 1), np.arange(ny + 1))
    d = rng.uniform(-0.1, 0.1, size=(2,) + i.shape)
    d[:, (i == 0) | (i == nx) | (j == 0) | (j == ny)] = 0.0
    xy = np.stack([(i + d[0]).ravel(), (j + d[1]).ravel()], 1) * h
    a = (np.arange(ny)[:, None] * (nx + 1) + np.arange(nx)[None, :]).ravel()
    tri = np.empty((2 * nx * ny, 3), dtype=np.int32)
    tri[0::2] = np.stack([a, a + 1, a + nx + 2], 1)
    tri[1::2] = np.stack([a, a + nx + 2, a + nx + 1], 1)
    return xy, tri


def _model(N, nx, ny, shots, nrcv, seed):
    """One seeded model: mesh, materials, sources, receivers, time step."""
    rng = np.random.default_rng([seed, N, nx, ny, shots, nrcv])
    h = 20.0
    xy, tri = _mesh(nx, ny, h, rng)
    ne = tri.shape[0]
    vp = VP * np.exp(rng.normal(0.0, 0.1, size=ne) - 0.005)
    vs = vp / math.sqrt(3.0)
    rho = np.full(ne, RHO)
    mu = rho * vs * vs
    lam = rho * vp * vp - 2.0 * mu
    top = ny * h
    # Shots in the upper element rows, receivers a third of an element deep.
    src = np.stack([rng.uniform(1.0, nx - 1.0, size=shots) * h, top - rng.uniform(0.3, 2.0, size=shots) * h], 1)
    rcv = np.stack([rng.uniform(0.5, nx - 0.5, size=nrcv) * h, np.full(nrcv, top - 0.34 * h)], 1)
    # About two fifths of the stability limit of this mesh family.
    dt = 0.12 * h / (vp.max() * N * N)
    f0 = VP / (6.0 * h)  # dominant P wavelength of six elements
    return dict(xy=xy, tri=tri, lam=lam, mu=mu, rho=rho, src=src, rcv=rcv, dt=dt, f0=f0, t0=1.0 / f0, N=N)


def _models(case, seed):
    if case["kind"] != "batch":
        return [_model(case["N"], case["nx"], case["ny"], case["shots"], case["nrcv"], seed)]
    rng = np.random.default_rng([1, case["meshes"], case["tri_min"], case["tri_max"]])  # the same sizes for every seed
    out = []
    for m in range(case["meshes"]):
        nsq = int(rng.integers(case["tri_min"], case["tri_max"] + 1)) // 2
        ny = max(4, int(round(math.sqrt(nsq / 2))))
        N = case["n_min"] + int(rng.integers(0, case["n_max"] - case["n_min"] + 1))
        out.append(_model(N, max(4, nsq // ny), ny, 1, case["nrcv"], seed * 1000 + m))
    return out


def _create(case, m):
    sim = capi.Simulation.create(m["xy"], m["tri"], m["N"], m["lam"], m["mu"], m["rho"], m["src"], m["rcv"],
                                 penalty=PENALTY, precision=case["precision"], op=case["op"])
    sim.set_dt(m["dt"])
    for s in range(len(m["src"])):
        sim.set_ricker(s, m["f0"], m["t0"], -1e9, 1, case["steps"] + 1)
    return sim


def prepare(case, seed):
    models = _models(case, seed)
    if case["kind"] == "survey":
        return dict(case=case, model=models[0])
    if case["kind"] == "batch":
        probs = []
        for m in models:
            src = [Source(x, y, m["f0"], m["t0"], -1e9, 1) for x, y in m["src"].tolist()]
            mesh = Mesh(m["xy"], m["tri"], np.ones(len(m["tri"]), dtype=np.int32), 0.0, 0.0)
            probs.append(Problem("mesh", mesh, m["N"], m["lam"], m["mu"], m["rho"], src, m["rcv"].tolist(),
                                 case["steps"], penalty=PENALTY))
        b = capi.Batch(probs, precision=case["precision"], op=case["op"])
        b.set_dt([m["dt"] for m in models])
        b.set_ricker(case["steps"] + 1)
        b.set_seismogram_capacity(case["steps"])
        b.first_step()
        return dict(case=case, batch=b, done=1)
    sim = _create(case, models[0])
    if case["kind"] == "run":
        sim.set_seismogram_capacity(case["steps"])
        sim.first_step()
    return dict(case=case, sim=sim)


def _kept(case, a):
    return a.astype(np.float32) if case["precision"] == "fp32" else a


# ------------------------------------------------------------------- pass --
def run(state):
    case = state["case"]
    steps = case["steps"]
    if case["kind"] == "run":
        sim = state["sim"]
        k0, _ = sim.progress()
        sim.run(steps)
        return dict(gather=_kept(case, sim.seismograms(k0, steps)), u=_kept(case, sim.u_all()))
    if case["kind"] == "batch":
        b, k0 = state["batch"], state["done"]
        b.run(steps)
        state["done"] += steps
        n = range(case["meshes"])
        return dict(gather=_kept(case, np.stack([b.seismograms(m, k0, steps) for m in n])),
                    u=_kept(case, np.concatenate([b.u(m) for m in n])))
    if case["kind"] == "cfl":
        return state["sim"].estimate_lmax(steps)
    sim = _create(case, state["model"])
    sim.set_seismogram_capacity(steps + 1)
    sim.first_step()
    sim.run(steps)
    out = dict(gather=_kept(case, sim.seismograms(0, steps + 1)), u=_kept(case, sim.u_all()))
    sim.close()
    return out


def _per_mesh(case):
    """(elements, blocks, modes per component) of each mesh of a case."""
    if case["kind"] != "batch":
        return [_counts(case["N"], case["nx"], case["ny"])]
    rng = np.random.default_rng([1, case["meshes"], case["tri_min"], case["tri_max"]])
    out = []
    for _ in range(case["meshes"]):
        nsq = int(rng.integers(case["tri_min"], case["tri_max"] + 1)) // 2
        ny = max(4, int(round(math.sqrt(nsq / 2))))
        N = case["n_min"] + int(rng.integers(0, case["n_max"] - case["n_min"] + 1))
        out.append(_counts(N, max(4, nsq // ny), ny))
    return out


def _counts(N, nx, ny):
    ne = 2 * nx * ny
    return ne, 4 * ne - 2 * (nx + ny), (N + 1) * (N + 2) // 2


def work(case):
    """One pass: per step the operator once (stored blocks; for the
    matrix-free form 25 values and 6 indices per element), u^k and u^{k-1}
    read and u^{k+1} written, plus the outputs handed back."""
    S, steps, nbytes, flops = case.get("shots", 1), case["steps"], 0.0, 0.0
    for ne, nnzb, Np in _per_mesh(case):
        R, N = 2 * Np, int(round((math.sqrt(8 * Np + 1) - 3) / 2))
        if case["op"] == "matrix_free":
            oper = ne * (25 * 8 + 6 * 4)
            f = ne * (2.0 * 4 * 2 * Np * Np + 3 * 2 * 2.0 * 2 * 3 * (N + 1) * Np)
        else:
            oper = nnzb * R * R * WEIGHT[case["precision"]]
            f = 2.0 * nnzb * R * R * S
        nbytes += steps * (oper + S * ne * R * (16 if case["kind"] == "cfl" else 24) + 8 * ne)
        flops += steps * f
        if case["kind"] != "cfl":
            nbytes += S * (ne * R + steps * case["nrcv"] * 2) * 8
    return {"bytes": nbytes, "flops": flops}


# ---------------------------------------------- the recurrence in 64 bits --
def _jacobi(n, a, b, z):
    p0, p1 = np.ones_like(z), 0.5 * (a - b + (a + b + 2.0) * z)
    if n == 0:
        return p0
    for k in range(2, n + 1):
        c = 2.0 * k + a + b
        p0, p1 = p1, ((c - 1.0) * (c * (c - 2.0) * z + a * a - b * b) * p1
                      - 2.0 * (k + a - 1.0) * (k + b - 1.0) * c * p0) / (2.0 * k * (k + a + b) * (c - 2.0))
    return p1


def _basis(N, x, y):
    """Orthonormal Dubiner polynomials of the reference triangle at (x, y):
    [points, modes], the second index outermost."""
    out = []
    for j in range(N + 1):
        for i in range(N + 1 - j):
            c = math.sqrt((2.0 * i + 1) * 2.0 * (i + j + 1))
            out.append(c * (1 - y) ** i * _jacobi(i, 0, 0, 2 * x / (1 - y) - 1) * _jacobi(j, 2 * i + 1, 0, 2 * y - 1))
    return np.stack(out, -1)


def _grad(N, x, y):
    """Gradients by the complex step (exact for polynomials): two arrays [points, modes]."""
    t = 1e-40
    return _basis(N, x + 1j * t, y + 0j).imag / t, _basis(N, x + 0j, y + 1j * t).imag / t


def _operator(m, dev):
    """The assembled operator and what the recurrence needs, on `dev`."""
    N, Q = m["N"], m["N"] + 1
    Np = Q * (Q + 1) // 2
    g, w = np.polynomial.legendre.leggauss(Q)
    # Volume rule on the collapsed square, edge rule on [0, 1].
    qx = ((1 + g[:, None]) / 2 + 0 * g[None, :]).ravel()
    qy = ((1 - g[:, None]) * (1 + g[None, :]) / 4).ravel()
    qw = ((1 - g[:, None]) * w[:, None] * w[None, :] / 8).ravel()
    G = _grad(N, qx, qy)
    K = np.stack([np.einsum("q,qi,qj->ij", qw, G[a], G[b]) for a in range(2) for b in range(2)])
    s, ws = (1 + g) / 2, w / 2
    ends = [(1 - s, s), (0 * s, 1 - s), (s, 0 * s)]  # edge l lies opposite vertex l
    Be = np.stack([_basis(N, *p) for p in ends])               # [3, Q, Np]
    Ge = np.stack([np.stack(_grad(N, *p)) for p in ends])      # [3, 2, Q, Np]

    T = lambda a: torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device=dev)  # noqa: E731
    tri = torch.as_tensor(m["tri"].astype(np.int64), device=dev)
    P = T(m["xy"])[tri]
    ne = tri.shape[0]
    J = torch.stack([P[:, 1] - P[:, 0], P[:, 2] - P[:, 0]], 2)
    det = J[:, 0, 0] * J[:, 1, 1] - J[:, 0, 1] * J[:, 1, 0]
    iJ = torch.linalg.inv(J)                                   # [e, reference a, physical p]
    # Neighbours: the directed edge (v, w) of one triangle is (w, v) of the other.
    va, vb = tri[:, [1, 2, 0]], tri[:, [2, 0, 1]]
    nv = int(tri.max()) + 1
    fwd, rev = (va * nv + vb).reshape(-1), (vb * nv + va).reshape(-1)
    order = torch.argsort(fwd)
    at = torch.searchsorted(fwd[order], rev).clamp(max=3 * ne - 1)
    mate = torch.where(fwd[order][at] == rev, order[at], torch.full_like(at, -1)).reshape(ne, 3)
    d = P[:, [2, 0, 1]] - P[:, [1, 2, 0]]                      # along edge l
    L = d.norm(dim=2)
    nrm = torch.stack([d[:, :, 1], -d[:, :, 0]], 2) / L[:, :, None]

    lam, mu, rho = T(m["lam"]), T(m["mu"]), T(m["rho"])
    eye = torch.eye(2, dtype=torch.float64, device=dev)
    # Hooke's law: C[e, m, k, n, l] d_l u_n contracted to sigma_mk.
    C = (lam[:, None, None, None, None] * torch.einsum("mk,nl->mknl", eye, eye)
         + mu[:, None, None, None, None] * (torch.einsum("mn,kl->mknl", eye, eye) + torch.einsum("ml,kn->mknl", eye, eye)))
    Kt, Bt, Gt, W = T(K.reshape(2, 2, Np, Np)), T(Be), T(Ge), T(ws)
    blocks = torch.zeros(ne, 2, Np, 4, 2, Np, dtype=torch.float64, device=dev)
    alpha = torch.einsum("emknl,eak,ebl->emnab", C, iJ, iJ) * det.abs()[:, None, None, None, None]
    blocks[:, :, :, 0] = torch.einsum("emnab,abij->eminj", alpha, Kt)
    # Traction of u on face l: t_m = sum_na beta[e, l, m, n, a] (d_a u_n).
    beta = torch.einsum("emknl,efk,eal->efmna", C, nrm, iJ)
    har = lambda a, b: 2 * a * b / (a + b)  # noqa: E731
    for l in range(3):
        for lp in range(3):
            e = torch.nonzero((mate[:, l] >= 0) & (mate[:, l] % 3 == lp))[:, 0]
            if not len(e):
                continue
            f = mate[e, l] // 3
            n = nrm[e, l]
            hl, hm = har(lam[e], lam[f]), har(mu[e], mu[f])
            # Penalty matrix of the face from harmonic means.
            c = torch.empty(len(e), 2, 2, dtype=torch.float64, device=dev)
            c[:, 0, 0] = (hl + 2 * hm) * n[:, 0] ** 2 + 2 * hm * n[:, 1] ** 2
            c[:, 1, 1] = (hl + 2 * hm) * n[:, 1] ** 2 + 2 * hm * n[:, 0] ** 2
            c[:, 0, 1] = c[:, 1, 0] = hl * n[:, 0] * n[:, 1]
            c *= PENALTY * N * N
            half = 0.5 * L[e, l, None, None, None]
            be, bf = beta[e, l] * half, beta[f, lp] * half
            Bs, Gs = Bt[l], Gt[l]
            Bn, Gn = Bt[lp].flip(0), Gt[lp].flip(1)            # the same points seen from the neighbour
            own = torch.einsum("enma,aqi,qj,q->eminj", be, Gs, Bs, W)  # traction of the test function
            blocks[e, :, :, 0] += (torch.einsum("emn,qi,qj,q->eminj", c, Bs, Bs, W)
                                   - own - own.permute(0, 3, 4, 1, 2))
            blocks[e, :, :, 1 + l] = (-torch.einsum("emn,qi,qj,q->eminj", c, Bs, Bn, W)
                                      + torch.einsum("enma,aqi,qj,q->eminj", be, Gs, Bn, W)
                                      + torch.einsum("emna,qi,aqj,q->eminj", bf, Bs, Gn, W))
    nb = torch.cat([torch.arange(ne, device=dev)[:, None], torch.where(mate >= 0, mate // 3, 0)], 1)
    return blocks.reshape(ne, 2 * Np, 8 * Np), nb, 1.0 / (rho * det), P[:, 0], iJ


def _point(m, op, pts, dev):
    """Elements and basis values of points: the first triangle that holds each."""
    _, _, _, p0, iJ = op
    el, ph = [], []
    for x in torch.as_tensor(pts, dtype=torch.float64, device=dev):
        r = torch.einsum("eak,ek->ea", iJ, x[None] - p0)
        e = int(torch.nonzero((r.min(1).values >= -1e-6) & (r.sum(1) <= 1 + 1e-6))[0, 0])
        rx, ry = r[e].tolist()
        el.append(e)
        ph.append(_basis(m["N"], np.array([rx]), np.array([ry]))[0])
    return torch.tensor(el, device=dev), torch.as_tensor(np.array(ph), device=dev)


def _exact_model(m, steps, nrcv, dev):
    """Gather [shots, steps + 1, receivers, 2] and final u [shots, unknowns] after first_step and `steps` steps."""
    op = _operator(m, dev)
    B, nb, minv = op[:3]
    ne, R = B.shape[0], B.shape[1]
    S, Np = len(m["src"]), R // 2
    se, sphi = _point(m, op, m["src"], dev)
    re, rphi = _point(m, op, m["rcv"], dev)
    dt, shots = m["dt"], torch.arange(S, device=dev)
    u = torch.zeros(ne, R, S, dtype=torch.float64, device=dev)
    up = torch.zeros_like(u)
    out, t = [], 0.0
    for k in range(steps + 1):
        a = math.pi ** 2 * m["f0"] ** 2 * (t - m["t0"]) ** 2
        F = -1e9 * (1 - 2 * a) * math.exp(-a)
        r = torch.bmm(B, u[nb].reshape(ne, 4 * R, S))
        r[se, Np:, shots] -= F * sphi  # all shots at once: one source row each
        r *= (-dt * dt * (0.5 if k == 0 else 1.0)) * minv[:, None, None]
        r += u if k == 0 else 2 * u - up
        up, u = u, r
        v = u[re].reshape(nrcv, 2, Np, S)
        out.append(torch.einsum("rcis,ri->src", v, rphi))
        t = t + dt if k else dt + dt
    gather = torch.stack(out, 1)
    return gather, u.reshape(ne, 2, Np, S).permute(3, 1, 0, 2).reshape(S, -1)


def exact(case, seed):
    if case["kind"] == "cfl":
        return None  # a Rayleigh quotient after a fixed number of iterations: no value of its own
    models = _models(case, seed)
    ne, nnzb, Np = max(_per_mesh(case))
    if nnzb * (2 * Np) ** 2 * 8 > 24e9 or work(case)["flops"] > 4e13:
        return None
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    got = [_exact_model(m, case["steps"], case["nrcv"], dev) for m in models]
    if case["kind"] == "survey":
        return dict(gather=got[0][0].cpu().numpy(), u=got[0][1].cpu().numpy())
    if case["kind"] == "batch":
        return dict(gather=np.stack([g[0, 1:].cpu().numpy() for g, _ in got]),
                    u=np.concatenate([u[0].cpu().numpy() for _, u in got]))
    return dict(gather=got[0][0][:, 1:].cpu().numpy(), u=got[0][1].cpu().numpy())
