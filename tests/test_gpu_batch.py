"""Multi-mesh batch (uneven sizes and degrees, one graph for all) against
the same meshes run one by one (GPU)."""
import numpy as np
import pytest

from helpers import rel
from tspeed_b200 import capi
from tspeed_b200 import workloads as W

pytestmark = pytest.mark.gpu


def small_batch():
    return W.mesh_batch(nmesh=6, seed=77, tri_range=(40, 160), N_range=(2, 5), nsteps=40)


@pytest.mark.parametrize("op,precision", [("explicit", "fp64"), ("matrix_free", "fp64"), ("explicit", "fp32")])
def test_batch_matches_single_meshes(op, precision):
    probs = small_batch()
    n = 40
    with capi.Batch(probs, precision=precision, op=op) as b:
        lmax = b.estimate_lmax(400)
        dt = 0.4 * 2 / np.sqrt(lmax)
        b.set_dt(dt)
        b.set_ricker(n)
        b.set_seismogram_capacity(n)
        b.first_step()
        b.run(17)
        b.run(n - 18)
        us = [b.u(m) for m in range(len(probs))]
        ss = [b.seismograms(m, 0, n) for m in range(len(probs))]
        assert b.ngroups == len(set(p.N for p in probs))
    tol = 1e-12 if precision == "fp64" else 1e-5
    for m, p in enumerate(probs):
        with capi.Simulation.from_problem(p, precision=precision, op=op) as s:
            l1 = s.estimate_lmax(400)
            assert abs(l1 - lmax[m]) / l1 < 1e-3  # different start vectors
            s.set_dt(dt[m])
            src = p.sources[0]
            s.set_ricker(0, src.f0, src.t0, src.amp, src.direction, n)
            s.first_step()
            s.run(n - 1)
            assert rel(us[m], s.u()) < tol
            assert rel(ss[m], s.seismograms(0, n)[0]) < tol


# The second shape's operator is above the size from which rows are claimed.
@pytest.mark.parametrize("N,nx,ny,op,precision", [(3, 30, 20, "matrix_free", "fp64"), (6, 60, 50, "explicit", "fp64"),
                                                  (6, 60, 100, "explicit", "fp32")])
def test_estimate_between_queued_steps_leaves_the_run_alone(N, nx, ny, op, precision):
    """Batch.run returns while its steps are queued; an estimate asked for then
    works on the same operators, edge values and row counters."""
    probs = []
    for i in range(2):
        m = W.jittered_rect(nx, ny, 20.0 * nx, 20.0 * ny, seed=i)
        lam, mu, rho = W.lame(np.full(m.ne, 3000.0), np.full(m.ne, 1700.0), np.full(m.ne, 2300.0))
        probs.append(W.Problem(str(i), m, N, lam, mu, rho, [W.Source(10.0 * nx + 1, 10.0 * ny + 1, 200.0, 1e-3, -1e9, 1)],
                               [(5.0 * nx, 19.0 * ny)], 900))
    out = []
    for estimate in (False, True):
        with capi.Batch(probs, precision=precision, op=op) as b:
            lmax = b.estimate_lmax(8)
            b.set_dt(np.full(2, 1e-5))
            b.set_ricker(900)
            b.set_seismogram_capacity(900)
            b.first_step()
            for n in (400, 300, 199):
                b.run(n)
                if estimate:
                    assert np.allclose(b.estimate_lmax(8), lmax, rtol=1e-10 if precision == "fp64" else 1e-5, atol=0)
            out.append([b.u(m) for m in range(2)] + [b.seismograms(m, 0, 900) for m in range(2)])
    assert all(np.any(u) for u in out[0][:2])
    for x, y in zip(*out):
        assert np.array_equal(x, y)


# Groups on both sides of the sizes between which matrix-free groups of a batch
# of three and more degrees are stepped by the lean kernel.
@pytest.mark.parametrize("nx,ny", [(10, 10), (17, 6), (25, 20), (21, 24)])
def test_matrix_free_batch_of_three_degrees(nx, ny):
    probs = []
    for N in (2, 4, 7):
        m = W.jittered_rect(nx, ny, 100.0 * nx, 100.0 * ny, seed=N)
        lam, mu, rho = W.lame(np.full(m.ne, 3000.0), np.full(m.ne, 1700.0), np.full(m.ne, 2300.0))
        probs.append(W.Problem(str(N), m, N, lam, mu, rho, [W.Source(51.0 * nx, 47.0 * ny, 200.0, 1e-3, -1e9, 1)],
                               [(52.0 * nx, 49.0 * ny), (50.0, 60.0)], 30))
    with capi.Batch(probs, op="matrix_free") as b:
        b.set_dt(np.full(3, 1e-4))
        b.set_ricker(30)
        b.first_step()
        b.run(29)
        out = [(b.u(i), b.seismograms(i, 0, 30)) for i in range(3)]
    for p, (u, seis) in zip(probs, out):
        with capi.Simulation.from_problem(p, op="matrix_free") as s:
            s.set_dt(1e-4)
            s.set_ricker(0, 200.0, 1e-3, -1e9, 1, 30)
            s.first_step()
            s.run(29)
            assert rel(u, s.u()) < 1e-12 and rel(seis, s.seismograms(0, 30)[0]) < 1e-12
