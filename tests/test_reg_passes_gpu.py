"""FP32 split-step passes on the register-resident transforms, every size along both axes,
against the FP64 oracle.

Tolerance: three steps make six (K-outer) to twelve one-axis transform pairs of at most log2(4096) =
12 rounded levels plus the local step; 250 roundings of 6e-8 adding as a random walk stay below
1e-6, adding up at worst below 1.5e-5."""
from __future__ import annotations

import numpy as np
import pytest

from tests.conftest import rel_l2
from tests.test_split_gpu import _case, _engine, _half_scales, _oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("potential", [False, True])
@pytest.mark.parametrize("ordering", ["cpu", "kouter"])
@pytest.mark.parametrize("ny,nx", [(64, 64), (64, 128), (128, 64), (256, 8), (8, 256), (512, 4), (4, 512),
                                    (1024, 64), (64, 1024), (2048, 16), (16, 2048), (4096, 8), (8, 4096)])
def test_every_size_matches_oracle(cuda_lib, ny, nx, ordering, potential):
    c = _case(nx=nx, ny=ny, seed=nx + 3 * ny, potential=potential)
    steps = 3
    eng = _engine(c, "single")
    eng.split_advance(0 if ordering == "cpu" else 1, 0, steps, _half_scales(c["dt"], 0, steps))
    psi, res = eng.get_state()
    eng.close()
    if ordering == "kouter":
        psi = np.fft.ifft2(psi.astype(np.complex128), axes=(-2, -1))
    psi_o, f_o = _oracle(c, ordering, steps, "single")
    assert rel_l2(psi, psi_o) < 1.5e-5
    assert rel_l2(res, f_o[0]) < 1.5e-5


@pytest.mark.parametrize("n", [64, 512, 1024])
def test_member_results_do_not_depend_on_the_batch(cuda_lib, n):
    c = _case(nx=n, ny=64, seed=n)
    outs = []
    for members in (1, 40):
        eng = _engine(c, "single", members=members)
        eng.split_advance(0, 0, 2, np.repeat(_half_scales(c["dt"], 0, 2), members, axis=2))
        outs.append(eng.get_state())
        eng.close()
    for m in (0, 39):
        assert np.array_equal(outs[1][0][m], outs[0][0][0]) and np.array_equal(outs[1][1][m], outs[0][1][0])
