"""Grids beyond the block counts of a launch along y and z, and rows beyond the widest window: each
takes a kernel that holds it, with the bits of a kernel named by the caller."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,members,precision,kernel", [
    (16, 1200000, 1, "double", 1), (16, 1200000, 1, "single", 1), (600000, 8, 1, "single", 1),
    (128, 4, 70000, "single", 2)])
def test_large_counts_step(cuda_lib, nx, ny, members, precision, kernel):
    from polarism_gb300.engine import MemberPhysics, RK4Engine

    outs = []
    rng = np.random.default_rng(5)
    psi = rng.random((members, 1, ny, nx), dtype=np.float32) + 1j * rng.random((members, 1, ny, nx), dtype=np.float32)
    res = rng.random((members, 1, ny, nx), dtype=np.float32)
    env = rng.random((ny, nx))
    for kind in (0, kernel):
        eng = RK4Engine(nx, ny, members, 0.8, 0.7, 1e-3, MemberPhysics(), precision)
        if kind:
            eng.set_kernel(kind)
        eng.set_pump(env.astype(eng.real))
        eng.set_state(psi.astype(eng.complex), res.astype(eng.real))
        eng.advance(0, 2, np.full((2, 3, members), 0.3))
        outs.append(eng.get_state())
        eng.close()
    assert np.array_equal(outs[0][0], outs[1][0]) and np.array_equal(outs[0][1], outs[1][1])
