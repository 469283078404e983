"""FP32 RK4 steps with the kernel left to the library against the streaming kernel, bit for bit.

Every kernel evaluates the same operations per site, so whichever one a grid gets (tiles, windows
closed on themselves or in bands, the full-width kernel, the streaming kernel) has to give the
streaming kernel's bits.  The sizes sit where the window and tile arithmetic can go wrong: grids
smaller than a halo, odd rows (single-element copies, a repeated last column), rows one site past
a window, narrow last bands, block ranges that cross members and bands, fewer rows than a fill."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _run(nx, ny, members, kernel, noise, potential, lasers, eta, reservoir="single", steps=4):
    from polarism_gb300.engine import MemberPhysics, RK4Engine

    rng = np.random.default_rng(nx * 1000 + ny)
    phys = MemberPhysics(g_I=0.0005, kinetic_relaxation_eta=eta)
    eng = RK4Engine(nx, ny, members, 0.8, 0.7, 1e-3, phys, "single", potential=potential, pump_terms=lasers,
                    reservoir=reservoir, pump_per_member=members > 1, potential_per_member=members > 1)
    if kernel:
        eng.set_kernel(kernel)
    per = (members, 1) if members > 1 else ()
    eng.set_pump(rng.random((lasers,) + per + (ny, nx)).astype(eng.real))
    if potential:
        pot = 0.2 * rng.standard_normal(per + (ny, nx))
        pot = pot - 0.01j * rng.random(pot.shape) if potential == 2 else pot
        eng.set_potential(pot.astype(eng.complex if potential == 2 else eng.real))
    if noise:
        eng.set_noise([5 + m for m in range(members)], phys.gamma_C, phys.R, 1.0, 1e-3 / (4 * 0.56))
    psi = 0.3 * (rng.standard_normal(eng.shape) + 1j * rng.standard_normal(eng.shape))
    eng.set_state(psi.astype(eng.complex), rng.random(eng.res_shape).astype(eng.real))
    scale = np.linspace(0.2, 0.4, steps * 3 * lasers * members)
    eng.advance(2 ** 32 - 1, steps,
                scale.reshape((steps, 3) + ((lasers,) if lasers > 1 else ()) + (members,)))
    out = eng.get_state()
    eng.close()
    return out


SIZES = [(4, 4, 1), (5, 9, 2), (33, 40, 2), (64, 64, 100), (250, 100, 9), (301, 201, 8), (512, 300, 5), (501, 400, 4),
         (513, 600, 2), (600, 500, 3), (777, 333, 3), (1000, 500, 2), (1023, 300, 3), (1024, 300, 4),
         (1025, 400, 2), (2050, 250, 2), (3001, 120, 2), (4096, 160, 1), (9000, 40, 1)]


@pytest.mark.parametrize("nx,ny,members", SIZES)
@pytest.mark.parametrize("noise,potential,lasers,eta", [(True, 0, 1, 0.0), (True, 1, 1, 0.0), (False, 2, 1, 0.02),
                                                        (False, 0, 1, 0.02), (True, 1, 2, 0.0)])
def test_automatic_kernel_is_bitwise_the_streaming_kernel(cuda_lib, nx, ny, members, noise, potential, lasers,
                                                          eta):
    auto = _run(nx, ny, members, 0, noise, potential, lasers, eta)
    stream = _run(nx, ny, members, 1, noise, potential, lasers, eta)
    assert np.array_equal(auto[0], stream[0]) and np.array_equal(auto[1], stream[1])


@pytest.mark.parametrize("nx,ny,members", [(9, 7, 3), (130, 90, 1), (255, 257, 2)])
@pytest.mark.parametrize("reservoir", ["double", "quadratic-double"])
def test_two_field_tiles_are_bitwise_the_streaming_kernel(cuda_lib, nx, ny, members, reservoir):
    auto = _run(nx, ny, members, 0, True, 1, 1, 0.0, reservoir)
    stream = _run(nx, ny, members, 1, True, 1, 1, 0.0, reservoir)
    assert np.array_equal(auto[0], stream[0]) and np.array_equal(auto[1], stream[1])
