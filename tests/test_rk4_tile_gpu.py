"""The RK4 tile kernel (the automatic choice in double precision) against the streaming kernel.

Both evaluate the same operations per site, so every tile shape, partial edge tile and wrap has
to give the streaming kernel's bits; the streaming kernel itself is held to the oracle and to the
reference's own trajectories elsewhere.  Sizes sit at the edges: grids smaller than one tile's
halo, one site over a tile, exact tiles, and one grid per tile shape the dispatch picks."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _run(nx, ny, members, kernel, noise, reservoir, potential, lasers, eta, precision="double", steps=3):
    from polarism_gb300.engine import MemberPhysics, RK4Engine

    rng = np.random.default_rng(nx * 1000 + ny)
    phys = MemberPhysics(g_I=0.0005, kinetic_relaxation_eta=eta)
    eng = RK4Engine(nx, ny, members, 0.8, 0.7, 1e-3, phys, precision, reservoir=reservoir, potential=potential,
                    pump_terms=lasers)
    if kernel:
        eng.set_kernel(kernel)
    eng.set_pump(rng.random((lasers, ny, nx)).astype(eng.real))
    if potential:
        pot = 0.2 * rng.standard_normal((ny, nx))
        pot = pot - 0.01j * rng.random((ny, nx)) if potential == 2 else pot
        eng.set_potential(pot.astype(eng.complex if potential == 2 else eng.real))
    if noise:
        eng.set_noise([5 + m for m in range(members)], phys.gamma_C, phys.R, 1.0, 1e-3 / (4 * 0.56))
    psi = 0.3 * (rng.standard_normal(eng.shape) + 1j * rng.standard_normal(eng.shape))
    eng.set_state(psi.astype(eng.complex), rng.random(eng.res_shape).astype(eng.real) if reservoir != "none" else None)
    eng.advance(7, steps, np.full((steps, 3) + ((lasers,) if lasers > 1 else ()) + (members,), 0.3))
    out = eng.get_state()
    eng.close()
    return out


@pytest.mark.parametrize("nx,ny,members", [(4, 4, 1), (5, 9, 2), (16, 8, 1), (17, 9, 1), (31, 70, 3),
                                            (33, 33, 1), (256, 256, 1), (230, 190, 8), (520, 1000, 1)])
@pytest.mark.parametrize("noise,reservoir,potential,lasers,eta", [
    (False, "single", 0, 1, 0.0), (True, "single", 0, 1, 0.0), (True, "single", 2, 2, 0.03),
    (True, "double", 1, 1, 0.0), (False, "quadratic-double", 0, 3, 0.0), (True, "none", 0, 1, 0.0)])
def test_tile_kernel_is_bitwise_the_streaming_kernel(cuda_lib, nx, ny, members, noise, reservoir, potential,
                                                     lasers, eta):
    tile = _run(nx, ny, members, 0, noise, reservoir, potential, lasers, eta)
    stream = _run(nx, ny, members, 1, noise, reservoir, potential, lasers, eta)
    assert np.array_equal(tile[0], stream[0])
    if reservoir != "none":
        assert np.array_equal(tile[1], stream[1])
