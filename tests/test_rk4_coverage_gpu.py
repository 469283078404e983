"""Every kernel and shape that the automatic choice takes on an FP32 grid, against the streaming kernel, bit
for bit, with the choice asserted so that a later fit of it cannot quietly leave a kernel untested.

The windows sit where their arithmetic can go wrong: each capacity closed on itself and in bands, on even and
odd rows, with blocks that cross members."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from tests.test_rk4_routes_gpu import _run

pytestmark = pytest.mark.gpu

OPTIONS = [(False, 0, 1, 0.0), (True, 0, 1, 0.02), (True, 1, 1, 0.0), (False, 2, 1, 0.02), (True, 2, 1, 0.0),
           (True, 0, 2, 0.0)]


def _plan(lib, nx, ny, members, noise, potential, lasers, eta):
    import torch

    from polarism_gb300 import _lib

    cfg = _lib.PgConfig(nx=nx, ny=ny, members=members, precision=_lib.PG_SINGLE, reservoir=1, potential=potential,
                        dx=0.8, dy=0.7, dt=1e-3, components=1, reservoir_components=1, pump_terms=lasers)
    plan = (C.c_int32 * 4)()
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    _lib.check(lib.pg_rk4_plan(C.byref(cfg), int(eta > 0), int(noise), sms, plan), "pg_rk4_plan")
    return list(plan)


@pytest.mark.parametrize("nx,ny,members,capacity,bands", [
    (640, 300, 4, 1024, 1), (637, 347, 3, 1024, 1), (1019, 300, 6, 1024, 1), (2028, 247, 4, 1024, 2),
    (2277, 742, 1, 1024, 3), (600, 500, 3, 320, 2), (3000, 100, 2, 512, 7)])
@pytest.mark.parametrize("noise,potential,lasers,eta", OPTIONS)
def test_windows(cuda_lib, nx, ny, members, capacity, bands, noise, potential, lasers, eta):
    plan = _plan(cuda_lib, nx, ny, members, noise, potential, lasers, eta)
    assert plan[:3] == [5, capacity, bands]
    auto = _run(nx, ny, members, 0, noise, potential, lasers, eta)
    stream = _run(nx, ny, members, 1, noise, potential, lasers, eta)
    assert np.array_equal(auto[0], stream[0]) and np.array_equal(auto[1], stream[1])


def test_every_shape_is_chosen(cuda_lib):
    grids = [(nx, ny, m) for nx in (64, 100, 128, 256, 301, 512, 640, 1024, 2028, 3000) for ny in (16, 100, 300, 1024)
             for m in (1, 2, 4, 16, 64)]
    seen = set()
    for g in grids:
        for o in OPTIONS:
            plan = _plan(cuda_lib, *g, *o)
            seen.add(tuple(plan[:2]) if plan[0] in (4, 5) else (plan[0],))
    assert {(1,), (2,), (4, 0), (4, 1), (4, 2), (4, 3), (5, 256), (5, 320), (5, 512), (5, 1024)} <= seen


@pytest.mark.parametrize("nx,ny,members", [(64, 16, 1), (128, 128, 4), (256, 256, 2), (100, 100, 16), (512, 300, 1)])
@pytest.mark.parametrize("noise,potential,lasers,eta", OPTIONS)
def test_tiles(cuda_lib, nx, ny, members, noise, potential, lasers, eta):
    assert _plan(cuda_lib, nx, ny, members, noise, potential, lasers, eta)[0] in (4, 5)
    auto = _run(nx, ny, members, 0, noise, potential, lasers, eta)
    stream = _run(nx, ny, members, 1, noise, potential, lasers, eta)
    assert np.array_equal(auto[0], stream[0]) and np.array_equal(auto[1], stream[1])
