"""Kernels on symmetric block storage and the matrix-free tiles at the sizes
where they can go wrong (GPU), against the oracle's products and recurrence.

Tolerances: FP64 paths differ from the oracle in summation order only,
1e-13 of the result's norm for a product and 1e-12 over a few steps. FP32
operators hold each entry to 2^-24 of itself and, with one shot, sum at most
4 * 90 FP32 products per row: 360 * 2^-24 = 2.2e-5 bounds the relative error
of rows without cancellation; 1e-4 covers the few steps taken here."""
import ctypes

import numpy as np
import pytest

import tsp_oracle as O
from helpers import rel
from tspeed_b200 import capi
from tspeed_b200 import workloads as W

pytestmark = pytest.mark.gpu


def random_operator(ne, N, seed, symmetric):
    """A block-CSR operator on a random graph of degree 0..3 (rows of 1..4
    blocks, diagonal first); symmetric: block (f, e) is the transpose of
    (e, f), else every block is its own."""
    rng = np.random.default_rng(seed)
    R = (N + 1) * (N + 2)
    nb = [[] for _ in range(ne)]
    for e in range(ne):
        for f in rng.permutation(ne)[:6]:
            if f != e and f not in nb[e] and len(nb[e]) < 3 and len(nb[f]) < 3:
                nb[e].append(int(f))
                nb[int(f)].append(e)
    row_ptr, col, blocks = [0], [], []
    at = {}
    for e in range(ne):
        for f in [e] + nb[e]:
            B = rng.uniform(0.5, 1.0, size=(R, R)) / R
            if symmetric and f == e:
                B = 0.5 * (B + B.T)
            if symmetric and f < e:
                B = blocks[at[(f, e)]].T
            at[(e, f)] = len(col)
            col.append(f)
            blocks.append(np.ascontiguousarray(B))
        row_ptr.append(len(col))
    minv = rng.uniform(0.5, 2.0, size=ne)
    return np.array(row_ptr, np.int32), np.array(col, np.int32), np.array(blocks), minv


# One row, rows without neighbours, fewer rows than teams, and more rows than
# one round of teams; every degree that the ring kernel takes and one below.
@pytest.mark.parametrize("symmetric", [True, False])
@pytest.mark.parametrize("N,ne", [(2, 40), (3, 1), (3, 700), (4, 61), (5, 2), (5, 601), (6, 37), (7, 9), (8, 33)])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_single_shot_blocks(N, ne, symmetric, precision):
    row_ptr, col, blocks, minv = random_operator(ne, N, 7 * N + ne, symmetric)
    Np = (N + 1) * (N + 2) // 2
    rng = np.random.default_rng(ne)
    u0, v0 = rng.standard_normal((2, 2 * ne * Np))
    phi = rng.standard_normal((3, Np))
    rcv = [0, ne // 2, ne - 1]
    F = rng.standard_normal((4, 2))
    with capi.Simulation.from_blocks(row_ptr, col, blocks, minv, [ne - 1], phi[:1], rcv, phi, precision=precision) as s:
        y = s.apply(u0)
        assert rel(s.export_operator()[2], blocks) < (1e-15 if precision == "fp64" else 1e-7)
        s.set_dt(0.01)
        s.set_force_table(0, F)
        s.set_initial(0, u0, v0)
        s.first_step()
        s.step()
        s.run(2)
        u, seis = s.u(), s.seismograms(0, 4)[0]
    tol = (1e-13, 1e-12) if precision == "fp64" else (1e-4, 1e-4)
    assert rel(y, O.apply_B(row_ptr, col, blocks, u0, ne, Np)) < tol[0]
    ur, sr, _ = O.leapfrog(row_ptr, col, blocks, minv, ne, Np, 0.01, 4, ne - 1, phi[0], F, rcv, phi, u0, v0)
    assert rel(u, ur) < tol[1]
    assert rel(seis, sr) < tol[1]


# Shot counts at the edges of the 8-, 16-, 24- and 32-shot tiles and of one, two and three tiles.
@pytest.mark.parametrize("N,S", [(3, 2), (3, 8), (3, 33), (4, 9), (4, 65), (5, 16), (5, 17), (5, 24), (6, 25), (6, 48),
                                 (7, 32), (7, 70), (8, 3), (8, 24)])
@pytest.mark.parametrize("symmetric", [True, False])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_few_shots(N, S, symmetric, precision, monkeypatch):
    monkeypatch.delenv("TSP_BATCHED_VARIANT", raising=False)
    ne = 11
    row_ptr, col, blocks, minv = random_operator(ne, N, N + S, symmetric)
    Np = (N + 1) * (N + 2) // 2
    rng = np.random.default_rng(S)
    u0 = rng.standard_normal((S, 2 * ne * Np))
    sphi = rng.standard_normal((S, Np))
    se = rng.integers(0, ne, size=S)
    rphi = rng.standard_normal((2, Np))
    rcv = [4, 4]
    F = rng.standard_normal((S, 3, 2))
    with capi.Simulation.from_blocks(row_ptr, col, blocks, minv, se, sphi, rcv, rphi, precision=precision) as s:
        y = s.apply(u0[0])
        s.set_dt(0.01)
        for k in range(S):
            s.set_force_table(k, F[k])
            s.set_initial(k, u0[k])
        s.first_step()
        s.run(2)
        u, seis = s.u_all(), s.seismograms(0, 3)
    tol = (1e-13, 1e-12) if precision == "fp64" else (1e-4, 1e-4)
    assert rel(y, O.apply_B(row_ptr, col, blocks, u0[0], ne, Np)) < tol[0]
    for k in range(S):
        ur, sr, _ = O.leapfrog(row_ptr, col, blocks, minv, ne, Np, 0.01, 3, int(se[k]), sphi[k], F[k], rcv, rphi, u0[k])
        assert rel(u[k], ur) < tol[1]
        assert rel(seis[k], sr) < tol[1]


# Rows whose diagonal block is not the first, and rows without one: u^k of the
# update has its own way there.
@pytest.mark.parametrize("N,S", [(3, 9), (4, 24), (7, 6)])
@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_few_shots_without_diagonal(N, S, precision, monkeypatch):
    monkeypatch.delenv("TSP_BATCHED_VARIANT", raising=False)
    ne, Np = 12, (N + 1) * (N + 2) // 2
    row_ptr, col, blocks, minv = random_operator(ne, N, N + S, False)
    rp, keep = [0], []
    for e in range(ne):
        r = list(range(row_ptr[e], row_ptr[e + 1]))
        if len(r) > 1:
            r = r[1:] if e % 3 == 0 else r[1:] + r[:1] if e % 3 == 1 else r
        keep += r
        rp.append(len(keep))
    row_ptr, col, blocks = np.array(rp, np.int32), col[keep], blocks[keep]
    rng = np.random.default_rng(S)
    u0 = rng.standard_normal((S, 2 * ne * Np))
    phi = rng.standard_normal((S, Np))
    F = rng.standard_normal((S, 3, 2))
    with capi.Simulation.from_blocks(row_ptr, col, blocks, minv, [5] * S, phi, [4], phi[:1], precision=precision) as s:
        s.set_dt(0.01)
        for k in range(S):
            s.set_force_table(k, F[k])
            s.set_initial(k, u0[k])
        s.first_step()
        s.run(2)
        u = s.u_all()
    for k in range(S):
        ur, _, _ = O.leapfrog(row_ptr, col, blocks, minv, ne, Np, 0.01, 3, 5, phi[k], F[k], [4], phi[:1], u0[k])
        assert rel(u[k], ur) < (1e-12 if precision == "fp64" else 1e-4)


# Element counts around the tile of eight, and more tiles than one round of warps.
@pytest.mark.parametrize("N", range(1, 9))
@pytest.mark.parametrize("nx,ny", [(1, 1), (3, 1), (2, 2), (3, 3), (5, 5), (60, 57)])
def test_matrix_free_tiles(N, nx, ny):
    if nx == 60 and N > 4:
        nx, ny = 31, 29
    m = W.jittered_rect(nx, ny, 100.0 * nx, 100.0 * ny, seed=N)
    rng = np.random.default_rng(N)
    vp = 2500 + 1500 * rng.random(m.ne)
    lam, mu, rho = W.lame(vp, vp / 1.8, 2000 + 500 * rng.random(m.ne))
    out = {}
    x = rng.standard_normal(m.ne * (N + 1) * (N + 2))
    for op in ("explicit", "matrix_free"):
        with capi.Simulation.create(m.xy, m.tri, N, lam, mu, rho, [(40.0, 30.0)], [(61.0, 33.0), (20.0, 55.0)],
                                    penalty=10.0, op=op) as s:
            y = s.apply(x)
            lmax = s.estimate_lmax(20)
            s.set_dt(0.3 * 2 / np.sqrt(lmax) if op == "explicit" else out["explicit"][4])
            dt = 0.3 * 2 / np.sqrt(lmax)
            s.set_ricker(0, 20.0, 0.05, -1e9, 1, 20)
            s.set_initial(0, 1e-3 * x)
            s.enable_energy(True)
            s.first_step()
            s.run(9)
            s.apply(x)  # a product between steps leaves the state's edge values alone
            s.run(6)
            out[op] = (y, s.u(), s.seismograms(0, 16), s.energy(1, 15), dt, lmax)
    a, b = out["matrix_free"], out["explicit"]
    assert rel(a[0], b[0]) < 1e-13
    assert abs(a[5] - b[5]) < 1e-12 * b[5]
    for i in (1, 2, 3):
        assert rel(a[i], b[i]) < 1e-11


# Operators just below and above the size from which the teams claim their rows
# (more rows than the teams' first ones either way), against the matrix-free
# operator (bounds as above and in test_matrix_free_tiles).
@pytest.mark.parametrize("N,nx,ny,precision", [(6, 70, 70, "fp64"), (6, 76, 75, "fp64"), (6, 100, 60, "fp32"),
                                               (6, 112, 100, "fp32"), (7, 80, 75, "fp32"), (7, 84, 80, "fp32"),
                                               (8, 64, 60, "fp32"), (8, 68, 64, "fp32")])
def test_claimed_rows(N, nx, ny, precision):
    m = W.jittered_rect(nx, ny, 100.0 * nx, 100.0 * ny, seed=N)
    rng = np.random.default_rng(N)
    vp = 2500 + 1500 * rng.random(m.ne)
    lam, mu, rho = W.lame(vp, vp / 1.8, 2000 + 500 * rng.random(m.ne))
    x = rng.standard_normal(m.ne * (N + 1) * (N + 2))
    out = []
    for op, prec in (("matrix_free", "fp64"), ("explicit", precision)):
        with capi.Simulation.create(m.xy, m.tri, N, lam, mu, rho, [(40.0, 30.0)], [(61.0, 33.0), (20.0, 55.0)],
                                    penalty=10.0, op=op, precision=prec) as s:
            s.set_dt(1e-5)
            s.set_ricker(0, 20.0, 0.05, -1e9, 1, 20)
            y, lmax = s.apply(x), s.estimate_lmax(10)
            s.set_initial(0, 1e-3 * x)
            s.enable_energy(True)
            s.first_step()
            s.run(9)
            out.append((y, s.u(), s.seismograms(0, 10), s.energy(1, 9), lmax))
    a, b = out
    tol = 1e-11 if precision == "fp64" else 1e-4
    for i in range(4):
        assert rel(b[i], a[i]) < tol
    assert abs(b[4] - a[4]) < tol * a[4]


def test_large_read_back_matches_small_ones():
    """Copies of several megabytes pass through the pinned pieces, small ones
    do not: wrapped seismogram rings with rows above one 8 MiB piece, many
    rows per piece, and a whole wavefield of several shots."""
    m = W.jittered_rect(40, 40, 4000.0, 4000.0, seed=3)
    lam, mu, rho = W.lame(np.full(m.ne, 3000.0), np.full(m.ne, 1700.0), np.full(m.ne, 2300.0))
    shots = [(1000.0 + 37 * k, 3900.0) for k in range(6)]
    rcv = [(4000.0 * (r + 0.37) / 257, 3933.0) for r in range(257)]
    with capi.Simulation.create(m.xy, m.tri, 3, lam, mu, rho, shots, rcv, penalty=10.0) as s:
        s.set_dt(1e-4)
        for k in range(6):
            s.set_ricker(k, 20.0, 0.01, -1e9, 1, 3000)
        s.set_seismogram_capacity(2100)
        s.first_step()
        s.run(2999)  # the ring wraps inside [900, 3000)
        for k0, n in ((900, 2100), (1700, 300)):  # rows of 8.6 MB and of 1.2 MB
            big = s.seismograms(k0, n)
            small = np.concatenate([s.seismograms(k0 + i, min(15, n - i)) for i in range(0, n, 15)], axis=1)
            assert np.array_equal(big, small)
        u = s.u_all()
        for k in range(6):
            assert np.array_equal(u[k], s.u(k))


# Meshes on which every ring is refilled many times: a refill that overtakes
# the loads of the stage it replaces shows as a difference between two runs.
@pytest.mark.parametrize("N,nx,ny,S,precision", [(4, 80, 40, 1, "fp64"), (4, 80, 40, 8, "fp64"), (4, 121, 60, 24, "fp32"),
                                                 (3, 80, 40, 20, "fp64"), (8, 40, 30, 8, "fp32"), (5, 60, 40, 64, "fp64"),
                                                 (5, 60, 40, 64, "fp32"), (6, 80, 40, 1, "fp32")])
def test_repeated_steps_are_identical(N, nx, ny, S, precision, monkeypatch):
    # The batched kernels are pinned: two candidates of the autotuner may round differently.
    if S == 64:
        monkeypatch.setenv("TSP_BATCHED_VARIANT", "5" if precision == "fp64" else "8")
    else:
        monkeypatch.delenv("TSP_BATCHED_VARIANT", raising=False)
    m = W.jittered_rect(nx, ny, 20.0 * nx, 20.0 * ny, seed=N)
    lam, mu, rho = W.lame(np.full(m.ne, 3000.0), np.full(m.ne, 1700.0), np.full(m.ne, 2300.0))
    shots = [(20.0 * nx * (k + 0.5) / S, 10.0 * ny + 1.0) for k in range(S)]
    rng = np.random.default_rng(S)
    n = m.ne * (N + 1) * (N + 2)
    a, b = rng.standard_normal((2, n))
    with capi.Simulation.create(m.xy, m.tri, N, lam, mu, rho, shots, [], penalty=10.0, precision=precision) as s:
        s.set_dt(1e-6)
        u0, u1 = np.tile(a, (S, 1)), np.tile(b, (S, 1))
        ref = None
        for _ in range(12):
            s.set_state(u0, u1, 1, 1e-6)
            s.run(3)
            u = s.u_all()
            ref = u if ref is None else ref
            assert np.array_equal(u, ref)
        # Every shot had the same state and no force: every shot the same result.
        assert np.array_equal(ref, np.tile(ref[0], (S, 1)))


def test_window_of_seismogram_rings_above_2_gib():
    """The shots' rings lie further apart than the largest pitch of a 2-D copy."""
    m = W.jittered_rect(6, 5, 600.0, 500.0, seed=3)
    lam, mu, rho = W.lame(np.full(m.ne, 3000.0), np.full(m.ne, 1700.0), np.full(m.ne, 2300.0))
    rcv = [(600.0 * (r + 0.5) / 1500, 490.0) for r in range(1500)]
    out = []
    for cap in (16, 90000):
        with capi.Simulation.create(m.xy, m.tri, 3, lam, mu, rho, [(210.0, 480.0), (390.0, 480.0)], rcv,
                                    penalty=10.0) as s:
            s.set_dt(1e-4)
            for k in range(2):
                s.set_ricker(k, 200.0, 1e-3, -1e9, 1, 16)
            s.set_seismogram_capacity(cap)
            s.first_step()
            s.run(15)
            out.append(s.seismograms(4, 12))
    assert np.any(out[0][0]) and np.any(out[0][1]) and np.array_equal(*out)


def test_read_back_without_device_memory():
    """A wavefield is read without a transposed copy where the device has no
    room for one; the calls after it do not see the failed allocation."""
    rt = ctypes.CDLL("libcudart.so.12")
    m = W.jittered_rect(260, 260, 2600.0, 2600.0, seed=3)  # 135,200 triangles: 97 MB of displacements
    lam, mu, rho = W.lame(np.full(m.ne, 3000.0), np.full(m.ne, 1700.0), np.full(m.ne, 2300.0))
    ballast = []
    with capi.Simulation.create(m.xy, m.tri, 8, lam, mu, rho, [(1310.0, 1290.0)], [(1310.0, 1295.0)], penalty=10.0,
                                op="matrix_free") as s:
        s.set_dt(1e-6)
        s.set_ricker(0, 200.0, 0.0, -1e9, 1, 16)
        s.first_step()
        s.step()
        s.run(2)
        u0 = s.u()
        try:
            capi.release_cached_memory(0)
            for size in (1 << 30, 64 << 20, 4 << 20):
                p = ctypes.c_void_p()
                while rt.cudaMalloc(ctypes.byref(p), ctypes.c_size_t(size)) == 0:
                    ballast.append(ctypes.c_void_p(p.value))
            rt.cudaGetLastError()
            assert np.array_equal(s.u(), u0)
            s.step()
            s.run(2)
            u1 = s.u()
        finally:
            for p in ballast:
                rt.cudaFree(p)
        assert len(ballast) > 0 and np.array_equal(s.u(), u1) and not np.array_equal(u1, u0)


# Receivers in one element and over neighbouring ones, around the counts at
# which a warp turns from one receiver at a time to one per lane, and above 32.
@pytest.mark.parametrize("per_element", [1, 3, 4, 5, 31, 33, 70])
@pytest.mark.parametrize("N,precision,op", [(n, "fp64", "matrix_free") for n in range(1, 9)] +
                         [(n, "fp64", "explicit") for n in range(3, 9)] + [(n, "fp32", "explicit") for n in range(5, 9)])
def test_receivers_sample_their_element(N, precision, op, per_element):
    m = W.jittered_rect(5, 3, 500.0, 300.0, seed=N)
    lam, mu, rho = W.lame(np.full(m.ne, 3000.0), np.full(m.ne, 1700.0), np.full(m.ne, 2300.0))
    rng = np.random.default_rng(per_element)
    rcv = []
    for e in (2, 3, 4, 5, 17, m.ne - 1):  # a tile of eight elements, one alone, the last
        a, b, c = m.xy[m.tri[e]]
        for _ in range(per_element if e != 4 else 1):
            s, t = rng.uniform(0.1, 0.45, 2)
            rcv.append(tuple(a + s * (b - a) + t * (c - a)))
    rng.shuffle(rcv)
    Np = (N + 1) * (N + 2) // 2
    with capi.Simulation.create(m.xy, m.tri, N, lam, mu, rho, [(210.0, 140.0)], rcv, penalty=10.0, precision=precision,
                                op=op) as sim:
        sim.set_dt(1e-6)
        sim.set_initial(0, rng.standard_normal(2 * m.ne * Np))
        sim.first_step()
        sim.run(2)
        u, seis = sim.u().reshape(2, m.ne, Np), sim.seismograms(2, 1)[0, 0]
        _, _, elem, phi = sim.export_points()
    ref = np.einsum("ri,cri->rc", phi, u[:, elem])
    assert len(set(elem)) == 6
    assert rel(seis, ref) < 1e-13


# Sizes on both sides of the lines between kernels that lie on the number of
# triangles: the row and the ring kernel at N = 3, few-shot and batched kernels
# at N = 6, against the matrix-free operator.
@pytest.mark.parametrize("N,nx,ny,shots,precision", [(3, 62, 25, 1, "fp64"), (3, 47, 33, 1, "fp64"),
                                                     (3, 74, 25, 1, "fp64"), (3, 617, 3, 1, "fp64"),
                                                     (3, 70, 37, 1, "fp64"), (3, 72, 36, 1, "fp64"),
                                                     (3, 100, 60, 1, "fp64"), (3, 353, 17, 1, "fp64"),
                                                     (6, 50, 50, 33, "fp32"), (6, 51, 50, 33, "fp32")])
def test_lines_between_kernels_on_size(N, nx, ny, shots, precision, monkeypatch):
    monkeypatch.delenv("TSP_BATCHED_VARIANT", raising=False)
    m = W.jittered_rect(nx, ny, 100.0 * nx, 100.0 * ny, seed=N)
    rng = np.random.default_rng(N)
    vp = 2500 + 1500 * rng.random(m.ne)
    lam, mu, rho = W.lame(vp, vp / 1.8, 2000 + 500 * rng.random(m.ne))
    x = rng.standard_normal(m.ne * (N + 1) * (N + 2))
    out = []
    for op, prec, S in (("matrix_free", "fp64", 1), ("explicit", precision, shots)):
        with capi.Simulation.create(m.xy, m.tri, N, lam, mu, rho, [(40.0, 30.0)] * S, [(61.0, 33.0), (20.0, 55.0)],
                                    penalty=10.0, op=op, precision=prec) as s:
            s.set_dt(1e-5)
            y, lmax = s.apply(x), s.estimate_lmax(10)
            for k in range(S):
                s.set_ricker(k, 20.0, 0.05, -1e9, 1, 20)
                s.set_initial(k, 1e-3 * x)
            s.first_step()
            s.run(9)
            out.append((y, s.u(S - 1), s.seismograms(0, 10)[S - 1], lmax))
    a, b = out
    tol = 1e-11 if precision == "fp64" else 1e-4
    for i in range(3):
        assert rel(b[i], a[i]) < tol
    assert abs(b[3] - a[3]) < tol * a[3]


@pytest.mark.parametrize("N", range(1, 9))
def test_matrix_free_with_little_device_memory(N):
    """Where the edge values of the matrix-free tiles would take more than a
    quarter of the free memory, the handle steps without them."""
    rt = ctypes.CDLL("libcudart.so.12")
    rt.cudaMemGetInfo.argtypes = [ctypes.POINTER(ctypes.c_size_t)] * 2
    m = W.jittered_rect(200, 180, 2000.0, 1800.0, seed=N)
    kept = m.ne * (46 + 24 * (N + 1)) * 8  # 54 MB (N = 1) to 151 MB
    rng = np.random.default_rng(N)
    vp = 2500 + 1500 * rng.random(m.ne)
    lam, mu, rho = W.lame(vp, vp / 1.8, 2000 + 500 * rng.random(m.ne))
    x = rng.standard_normal(m.ne * (N + 1) * (N + 2))
    out, ballast = [], []
    try:
        for little in (False, True):
            if little:
                capi.release_cached_memory(0)
                room, total, p = ctypes.c_size_t(), ctypes.c_size_t(), ctypes.c_void_p()
                while True:
                    assert rt.cudaMemGetInfo(ctypes.byref(room), ctypes.byref(total)) == 0
                    spare = room.value - 3 * kept
                    if spare < (16 << 20) or rt.cudaMalloc(ctypes.byref(p), ctypes.c_size_t(min(spare, 1 << 30))) != 0:
                        break
                    ballast.append(ctypes.c_void_p(p.value))
                rt.cudaGetLastError()
            with capi.Simulation.create(m.xy, m.tri, N, lam, mu, rho, [(1010.0, 905.0)], [(1031.0, 933.0), (20.0, 55.0)],
                                        penalty=10.0, op="matrix_free") as s:
                y, lmax = s.apply(x), s.estimate_lmax(6)
                s.set_dt(1e-5)
                s.set_ricker(0, 20.0, 0.05, -1e9, 1, 20)
                s.set_initial(0, 1e-3 * x)
                s.enable_energy(True)
                s.first_step()
                s.run(9)
                out.append((y, s.u(), s.seismograms(0, 10), s.energy(1, 9), lmax))
    finally:
        for p in ballast:
            rt.cudaFree(p)
    a, b = out
    assert not np.array_equal(a[0], b[0])  # another kernel
    assert rel(b[0], a[0]) < 1e-13
    assert abs(b[4] - a[4]) < 1e-12 * a[4]
    for i in (1, 2, 3):
        assert rel(b[i], a[i]) < 1e-11


def test_reported_kernels(monkeypatch):
    """A forced number that names no FP32 batched kernel is reported as the
    kernel that runs; stored blocks tell symmetric storage from full."""
    m = W.jittered_rect(8, 5, 800.0, 500.0, seed=2)
    lam, mu, rho = W.lame(np.full(m.ne, 3000.0), np.full(m.ne, 1700.0), np.full(m.ne, 2300.0))
    nnzb = m.ne + 2 * ((3 * m.ne - 2 * (8 + 5)) // 2)

    def handle(N, shots, precision, op="explicit"):
        return capi.Simulation.create(m.xy, m.tri, N, lam, mu, rho, [(310.0 + k, 240.0) for k in range(shots)], [],
                                      penalty=10.0, precision=precision, op=op)
    for N, shown in ((4, 1), (6, 1), (7, 2)):
        monkeypatch.setenv("TSP_BATCHED_VARIANT", "14")
        with handle(N, 3, "fp32") as s:
            assert s.kernel_variant == shown and s.stored_blocks == s.nnzb == nnzb
    monkeypatch.delenv("TSP_BATCHED_VARIANT")
    half = m.ne + (nnzb - m.ne) // 2
    for N, shots, precision, op, stored in ((5, 1, "fp64", "explicit", half), (5, 3, "fp64", "explicit", half),
                                            (5, 3, "fp32", "explicit", half), (5, 64, "fp32", "explicit", nnzb),
                                            (2, 1, "fp64", "explicit", nnzb), (5, 1, "bf16", "explicit", nnzb),
                                            (5, 1, "fp64", "matrix_free", 0)):
        with handle(N, shots, precision, op) as s:
            assert s.nnzb == nnzb and s.stored_blocks == stored


# FP32 blocks of the few-shot kernel are widened and multiply the FP64 state:
# against the oracle on the rounded blocks only the order of FP64 sums differs
# (bounds as for FP64 blocks above).
@pytest.mark.parametrize("N,S", [(3, 2), (3, 32), (4, 9), (4, 24), (5, 16), (5, 24), (6, 25), (6, 48), (7, 32), (7, 70),
                                 (8, 3), (8, 24)])
def test_few_shots_of_fp32_blocks_sum_in_fp64(N, S, monkeypatch):
    monkeypatch.delenv("TSP_BATCHED_VARIANT", raising=False)
    ne, Np = 11, (N + 1) * (N + 2) // 2
    row_ptr, col, blocks, minv = random_operator(ne, N, N + S, True)
    rng = np.random.default_rng(S)
    u0 = rng.standard_normal((S, 2 * ne * Np))
    phi = rng.standard_normal((S, Np))
    F = rng.standard_normal((S, 3, 2))
    with capi.Simulation.from_blocks(row_ptr, col, blocks, minv, [5] * S, phi, [4], phi[:1], precision="fp32") as s:
        assert s.stored_blocks < s.nnzb
        s.set_dt(0.01)
        for k in range(S):
            s.set_force_table(k, F[k])
            s.set_initial(k, u0[k])
        s.first_step()
        s.run(2)
        u, seis = s.u_all(), s.seismograms(0, 3)
    rounded = blocks.astype(np.float32).astype(np.float64)
    for k in range(S):
        ur, sr, _ = O.leapfrog(row_ptr, col, rounded, minv, ne, Np, 0.01, 3, 5, phi[k], F[k], [4], phi[:1], u0[k])
        assert rel(u[k], ur) < 1e-12
        assert rel(seis[k], sr) < 1e-12


def test_single_shot_rows_in_any_order_at_a_size_line():
    """Rows whose diagonal block is not the first, at a size whose meshes take
    the row kernel (which reads u^k from the first block)."""
    N, ne, Np = 3, 3300, 10
    row_ptr, col, blocks, minv = random_operator(ne, N, 3, True)
    order = np.concatenate([np.roll(np.arange(row_ptr[e], row_ptr[e + 1]), e % 3) for e in range(ne)])
    col, blocks = col[order], blocks[order]
    rng = np.random.default_rng(7)
    u0 = rng.standard_normal(2 * ne * Np)
    phi = rng.standard_normal((1, Np))
    F = rng.standard_normal((3, 2))
    with capi.Simulation.from_blocks(row_ptr, col, blocks, minv, [9], phi, [ne - 1], phi) as s:
        s.set_dt(0.01)
        s.set_force_table(0, F)
        s.set_initial(0, u0)
        s.first_step()
        s.run(2)
        u = s.u()
    ur, _, _ = O.leapfrog(row_ptr, col, blocks, minv, ne, Np, 0.01, 3, 9, phi[0], F, [ne - 1], phi, u0)
    assert rel(u, ur) < 1e-12


# The row and the ring kernel for FP32 blocks at N = 3 and 4, on both sides of
# the sizes between them, against the matrix-free operator (bounds as above).
@pytest.mark.parametrize("N,nx,ny", [(3, 25, 20), (3, 51, 10), (4, 40, 40), (4, 59, 28), (4, 75, 50), (4, 94, 40)])
def test_fp32_rows_at_the_size_lines(N, nx, ny):
    m = W.jittered_rect(nx, ny, 100.0 * nx, 100.0 * ny, seed=N)
    rng = np.random.default_rng(N)
    vp = 2500 + 1500 * rng.random(m.ne)
    lam, mu, rho = W.lame(vp, vp / 1.8, 2000 + 500 * rng.random(m.ne))
    x = rng.standard_normal(m.ne * (N + 1) * (N + 2))
    out = []
    for op, prec in (("matrix_free", "fp64"), ("explicit", "fp32")):
        with capi.Simulation.create(m.xy, m.tri, N, lam, mu, rho, [(40.0, 30.0)], [(61.0, 33.0), (20.0, 55.0)],
                                    penalty=10.0, op=op, precision=prec) as s:
            s.set_dt(1e-5)
            y, lmax = s.apply(x), s.estimate_lmax(10)
            s.set_ricker(0, 20.0, 0.05, -1e9, 1, 20)
            s.set_initial(0, 1e-3 * x)
            s.first_step()
            s.run(9)
            out.append((y, s.u(), s.seismograms(0, 10), lmax))
            stored, nnzb = s.stored_blocks, s.nnzb
    rows = m.ne > 1000 if N == 3 else 3200 < m.ne <= 7500
    assert (stored == nnzb) == rows
    a, b = out
    for i in range(3):
        assert rel(b[i], a[i]) < 1e-4
    assert abs(b[3] - a[3]) < 1e-4 * a[3]
