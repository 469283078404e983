"""``RK4Engine.kernel()`` names the kernel that steps the grid, not one that could."""
from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nx,ny,members,precision,choice,eta,kernel", [
    (256, 256, 1, "single", 0, 0.0, 4),     # tiles, on a grid that the full-width kernel could take
    (1024, 8, 1, "single", 0, 0.0, 4),
    (600, 500, 3, "single", 0, 0.0, 5),     # windows
    (1024, 1024, 8, "single", 0, 0.0, 2),
    (64, 64, 128, "double", 0, 0.0, 4),
    (256, 256, 1, "single", 1, 0.0, 1),
    (1024, 64, 1, "single", 2, 0.0, 2),
    (1024, 64, 1, "single", 3, 0.0, 3),
    (1024, 64, 1, "single", 3, 0.02, 2)])   # four sites a thread has no relaxation: two run
def test_kernel_in_use(cuda_lib, nx, ny, members, precision, choice, eta, kernel):
    from polarism_gb300.engine import MemberPhysics, RK4Engine

    eng = RK4Engine(nx, ny, members, 0.8, 0.7, 1e-3, MemberPhysics(kinetic_relaxation_eta=eta), precision)
    if choice:
        eng.set_kernel(choice)
    assert eng.kernel() == kernel
    eng.close()
