"""A bounded wait that gave up is reported by every call that hands out what
the kernel wrote (GPU). The flag is set from the host: no wait runs out."""
import ctypes as C

import numpy as np
import pytest

from tspeed_b200 import capi
from tspeed_b200 import workloads as W

pytestmark = pytest.mark.gpu

TIMEOUT = -8


def model(seed=1):
    m = W.jittered_rect(6, 5, 600.0, 500.0, seed=seed)
    return m, W.lame(np.full(m.ne, 3000.0), np.full(m.ne, 1700.0), np.full(m.ne, 2300.0))


def noalloc(s):
    out = C.c_double()
    rc = capi.lib().tsp_estimate_lmax_noalloc(s._h, 3, C.byref(out))
    if rc:
        raise capi.TspError(rc, "")


def check(calls, flag):
    before = {name: call() for name, call in calls.items() if name not in ("run_timed", "estimate_lmax")}
    flag(1)
    for name, call in calls.items():
        with pytest.raises(capi.TspError) as e:
            call()
        assert e.value.code == TIMEOUT, name
    flag(0)
    # Nothing was written meanwhile.
    for name, old in before.items():
        if name != "noalloc":
            assert np.array_equal(np.asarray(calls[name]()), np.asarray(old)), name


@pytest.mark.parametrize("N,shots,precision", [(4, 1, "fp64"), (5, 1, "fp32"), (4, 3, "fp64"), (6, 3, "fp32")])
def test_simulation_calls_report_a_timeout(N, shots, precision, monkeypatch):
    monkeypatch.delenv("TSP_BATCHED_VARIANT", raising=False)
    m, (lam, mu, rho) = model()
    x = np.random.default_rng(N).standard_normal(m.ne * (N + 1) * (N + 2))
    with capi.Simulation.create(m.xy, m.tri, N, lam, mu, rho, [(310.0 + k, 240.0) for k in range(shots)],
                                W.surface_receivers(m, 3), penalty=10.0, precision=precision) as s:
        s.set_dt(1e-5)
        for k in range(shots):
            s.set_ricker(k, 20.0, 0.01, -1e9, 1, 20)
            s.set_initial(k, x)
        s.enable_energy(True)
        s.first_step()
        s.run(8)
        check({"u": s.u, "u_all": s.u_all, "seismograms": lambda: s.seismograms(0, 9), "energy": lambda: s.energy(1, 8),
               "get_state": lambda: s.get_state()[1], "check_finite": s.check_finite, "apply": lambda: s.apply(x),
               "noalloc": lambda: noalloc(s), "estimate_lmax": lambda: s.estimate_lmax(3),
               "field_values": s.field_values, "run_timed": lambda: s.run_timed(2)},
              lambda v: capi.lib().tsp_selftest_set_timeout(s._h, v))


@pytest.mark.parametrize("precision", ["fp64", "fp32"])
def test_batch_calls_report_a_timeout(precision):
    probs = []
    for N in (4, 5):
        m, (lam, mu, rho) = model(N)
        probs.append(W.Problem(str(N), m, N, lam, mu, rho, [W.Source(310.0, 240.0, 20.0, 0.01, -1e9, 1)],
                               W.surface_receivers(m, 3), 20))
    with capi.Batch(probs, precision=precision) as b:
        b.set_dt(np.full(2, 1e-5))
        b.set_ricker(20)
        b.set_seismogram_capacity(20)
        b.first_step()
        b.run(8)
        check({"u": lambda: b.u(1), "seismograms": lambda: b.seismograms(1, 0, 9),
               "estimate_lmax": lambda: b.estimate_lmax(3), "run_timed": lambda: b.run_timed(2)},
              lambda v: capi.lib().tsp_selftest_batch_set_timeout(b._b, v))
