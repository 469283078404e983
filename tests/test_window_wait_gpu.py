"""The bounded wait of the RK4 window kernel (one block an SM, complex potential): in the give-up setting
every wait on the block's barrier gives up at once, the failure is reported, the call returns, and the
same solver steps correctly afterwards."""
from __future__ import annotations

import ctypes as C
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,members,bands", [(640, 300, 4, 1), (637, 347, 3, 1), (2028, 247, 4, 2)])
def test_zero_poll_limit_reports_timeout_and_solver_recovers(cuda_lib, nx, ny, members, bands):
    import torch

    from polarism_gb300 import _lib
    from polarism_gb300.engine import MemberPhysics, RK4Engine

    rng = np.random.default_rng(nx)
    psi = (0.1 * (rng.standard_normal((members, 1, ny, nx)) + 1j * rng.standard_normal((members, 1, ny, nx)))
           ).astype(np.complex64)
    res = rng.random((members, 1, ny, nx)).astype(np.float32)
    env = rng.random((ny, nx)).astype(np.float32)
    pot = (0.1 * rng.standard_normal((ny, nx)) - 0.01j * rng.random((ny, nx))).astype(np.complex64)
    steps = 4
    scales = np.full((steps, 3, members), 0.05)

    def make(kind=0):
        eng = RK4Engine(nx, ny, members, 0.4, 0.4, 5e-4, MemberPhysics(), "single",
                        potential=_lib.PG_POT_COMPLEX)
        if kind:
            eng.set_kernel(kind)
        eng.set_pump(env)
        eng.set_potential(pot)
        eng.set_state(psi, res)
        return eng

    cfg = _lib.PgConfig(nx=nx, ny=ny, members=members, precision=_lib.PG_SINGLE, reservoir=1,
                        potential=_lib.PG_POT_COMPLEX, dx=0.4,
                        dy=0.4, dt=5e-4, components=1, reservoir_components=1, pump_terms=1)
    plan = (C.c_int32 * 4)()
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    _lib.check(cuda_lib.pg_rk4_plan(C.byref(cfg), 0, 0, sms, plan), "pg_rk4_plan")
    assert list(plan)[:3] == [5, 1024, bands]  # the capacity that has the split barrier
    eng = make()
    assert eng.kernel() == 5
    eng.set_wait_limit(0)
    t0 = time.perf_counter()
    eng.advance(0, steps, scales)
    status = eng.lib.pg_synchronize(eng.handle)
    elapsed = time.perf_counter() - t0
    assert status == _lib.PG_ERR_TIMEOUT, (status, eng.lib.pg_last_error())
    assert elapsed < 10.0, f"the failed advance took {elapsed:.1f} s"
    eng.set_wait_limit(100000)
    eng.set_state(psi, res)
    eng.advance(0, steps, scales)
    got = eng.get_state()
    eng.close()
    ref = make(1)
    ref.advance(0, steps, scales)
    want = ref.get_state()
    ref.close()
    assert np.array_equal(got[0], want[0]) and np.array_equal(got[1], want[1])
