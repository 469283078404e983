"""The automatic choice of RK4 kernel, computed without a GPU: every grid that some kernel takes gets a
kernel whose launch holds it (at most 65535 blocks along y and z, a row within a window)."""
from __future__ import annotations

import ctypes as C

import pytest


@pytest.fixture(scope="module")
def plan():
    from polarism_gb300 import _lib, build

    lib = _lib.load(build.build())

    def ask(nx, ny, members, precision="single", reservoir="single", potential=0, lasers=1, eta=False, noise=False, sms=152):
        cfg = _lib.PgConfig(nx=nx, ny=ny, members=members,
                            precision=_lib.PG_SINGLE if precision == "single" else _lib.PG_DOUBLE,
                            reservoir={"none": 0, "single": 1, "double": 2, "quadratic-double": 3}[reservoir],
                            potential=potential, dx=1.0, dy=1.0, dt=1e-3, components=1, reservoir_components=1,
                            pump_terms=lasers)
        out = (C.c_int32 * 4)()
        _lib.check(lib.pg_rk4_plan(C.byref(cfg), int(eta), int(noise), sms, out), "pg_rk4_plan")
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


@pytest.mark.parametrize("grid,options,noise,kernels", [
    # us a step of the kernels named against the ones that an estimate without the noise, the number of
    # schedulers or the crossings between members took
    ((128, 128, 128), {}, False, (WINDOW,)),                                 # 21.0; streaming 24.2
    ((64, 64, 64), {}, False, (STREAM,)),                                    # 7.9; tiles 8.9
    ((128, 128, 96), dict(potential=2), False, (WIDE,)),                     # 33.2; windows 39.0
    ((128, 128, 96), dict(potential=2), True, (WIDE,)),                      # 35.2; windows 42.9
    ((100, 100, 64), dict(potential=2), True, (STREAM,)),                    # 25.9; windows 32.7
    ((64, 64, 772), dict(eta=True), True, (STREAM,)),                        # 66.8; windows 102
    ((64, 64, 512), dict(lasers=2), True, (STREAM,)),                        # 74.8; windows 100
    ((64, 64, 1279), dict(lasers=2), False, (STREAM,)),                      # 140; windows 185
    ((600, 500, 6), dict(reservoir="double"), False, (STREAM,)),             # 65; tiles 77
    ((3000, 100, 2), dict(reservoir="none"), False, (STREAM,)),              # 23.6; tiles 27.9
    ((200, 200, 32), dict(potential=2), False, (WINDOW,)),                   # 30.9; streaming 47.9
    ((256, 256, 1), dict(lasers=2), False, (TILE,))])                        # 8.3; windows 9.6
def test_choice_follows_what_was_measured(plan, grid, options, noise, kernels):
    assert plan(*grid, noise=noise, **options)[0] in kernels


@pytest.mark.parametrize("grid,options,noise,kernel", [
    # us a step of the kernel named against the one that a coarser estimate took: warps that share the schedulers
    # unevenly, rows of 1024 sites, tiles by the round, the last wave of the streaming kernel's blocks
    ((1024, 741, 1), {}, True, WINDOW),                                      # 17.6; full width 20.0
    ((1024, 208, 4), {}, True, WINDOW),                                      # 18.6; full width 20.0
    ((4096, 133, 2), dict(potential=2), True, WINDOW),                       # 30.5; streaming 34.1
    ((163, 736, 7), {}, True, WINDOW),                                       # 20.0; streaming 22.2
    ((595, 93, 7), {}, True, WINDOW),                                        # 13.0; tiles 14.3
    ((137, 504, 6), dict(potential=2), True, WINDOW),                        # 23.5; streaming 25.4
    ((128, 128, 96), dict(potential=2), False, WIDE),                        # 33.0; streaming 37.5
    ((65, 65, 207), dict(potential=2), True, STREAM),                        # windows 20 % slower
    ((525, 954, 16), dict(reservoir="double"), False, STREAM)])              # 364; tiles 414
def test_choice_follows_warps_and_rounds(plan, grid, options, noise, kernel):
    assert plan(*grid, noise=noise, **options)[0] == kernel
