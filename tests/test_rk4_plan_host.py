"""The automatic choice of RK4 kernel, computed without a GPU: every grid that some kernel takes gets a
kernel whose launch holds it (at most 65535 blocks along y and z, a row within a window)."""
from __future__ import annotations

import ctypes as C

import pytest


@pytest.fixture(scope="module")
def plan():
    from polarism_gb300 import _lib, build

    lib = _lib.load(build.build())

    def ask(nx, ny, members, precision="single", reservoir="single", potential=0, lasers=1, eta=False, sms=152):
        cfg = _lib.PgConfig(nx=nx, ny=ny, members=members,
                            precision=_lib.PG_SINGLE if precision == "single" else _lib.PG_DOUBLE,
                            reservoir={"none": 0, "single": 1, "double": 2, "quadratic-double": 3}[reservoir],
                            potential=potential, dx=1.0, dy=1.0, dt=1e-3, components=1, reservoir_components=1,
                            pump_terms=lasers)
        out = (C.c_int32 * 4)()
        _lib.check(lib.pg_rk4_plan(C.byref(cfg), int(eta), sms, out), "pg_rk4_plan")
        return list(out)

    return ask


STREAM, WIDE, TILE, WINDOW = 1, 2, 4, 5
TILE_ROWS = (8, 16, 16, 32)


@pytest.mark.parametrize("precision", ["single", "double"])
@pytest.mark.parametrize("reservoir", ["none", "single", "double"])
@pytest.mark.parametrize("nx,ny,members", [
    (16, 1 << 20, 1), (16, (1 << 20) + 1, 1), (16, 1200000, 1), (4, 1 << 24, 1), (40, 3000000, 2), (4, 4, 65535),
    (1 << 20, 16, 1), (520000, 8, 1), (1 << 26, 4, 2), (256, 256, 1), (1024, 1024, 8)])
def test_launches_hold_the_grid(plan, nx, ny, members, precision, reservoir):
    kind, a, b, blocks = plan(nx, ny, members, precision, reservoir)
    if kind == STREAM:
        assert -(-ny // b) <= 65535 and members <= 65535
    elif kind == TILE:
        assert -(-ny // TILE_ROWS[a]) <= 65535 and members <= 65535
    else:
        assert precision == "single" and reservoir == "single"
        if kind == WINDOW:
            band = nx if b == 1 else -(-nx // b)
            assert a in (256, 320, 512, 1024) and 1 <= b <= nx and band + (8 if b > 1 else 0) <= a and blocks > 0


def test_more_members_than_a_launch_holds(plan):
    assert plan(128, 4, 70000)[0] in (WIDE, WINDOW)
    assert plan(100, 60, 100000)[0] == WINDOW
    assert plan(128, 4, 70000, reservoir="double")[0] == STREAM  # no kernel takes it: refused at the launch
