"""FP32 split-step passes on the register-resident transforms with every kind of local step: without
noise, without a reservoir, two-field reservoirs, several lasers, real potentials, in both orderings, against
the FP64 oracle.  Tolerance as for the single configuration (test_reg_passes_gpu.py): 250 roundings of
6e-8 stay below 1.5e-5 added up at worst."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import gpe
from tests.conftest import rel_l2

pytestmark = pytest.mark.gpu

P = dict(hbar=0.6582119514, m_eff=0.284, g_C=0.02, g_R=0.03, g_I=0.01, R=0.05, gamma_C=0.083, gamma_R=0.02,
         gamma_I=0.01, gamma_A=0.03, R_IA=0.05, R_AI=0.01, kappa=0.05)
OPTIONS = {
    "noise-free": dict(noise=False),
    "no-reservoir-real-potential": dict(kind="none", potential=1, noise=False),
    "double-noise": dict(kind="double"),
    "quadratic-double-two-lasers": dict(kind="quadratic-double", lasers=2, noise=False),
    "three-lasers-real-potential-noise": dict(lasers=3, potential=1),
}


@pytest.mark.parametrize("option", list(OPTIONS))
@pytest.mark.parametrize("ordering", ["cpu", "kouter"])
@pytest.mark.parametrize("ny,nx", [(64, 64), (128, 512), (256, 16), (8, 1024), (1024, 8), (2048, 8), (4, 4096)])
def test_local_steps_match_oracle(cuda_lib, ny, nx, ordering, option):
    from polarism_gb300.engine import Engine, MemberPhysics

    kind, lasers, potential, noise = (OPTIONS[option].get(k, d) for k, d in
                                      (("kind", "single"), ("lasers", 1), ("potential", 0), ("noise", True)))
    dx, dy, dt, steps = 1.1, 0.9, 0.01, 3
    rng = np.random.default_rng(nx + 3 * ny)
    psi0 = 0.5 * (rng.standard_normal((1, 1, ny, nx)) + 1j * rng.standard_normal((1, 1, ny, nx)))
    fields = tuple(rng.random((1, 1, ny, nx)) for _ in range({"none": 0, "single": 1}.get(kind, 2)))
    env = rng.random((lasers, ny, nx))
    pot = 0.05 * rng.standard_normal((ny, nx)) if potential else 0.0
    coeff = lambda l, t: 0.3 * (1 + 0.2 * l) * (1 + 0.4 * np.sin(30 * t + l))  # noqa: E731
    eng = Engine(nx, ny, 1, dx, dy, dt, MemberPhysics(**P), "single", reservoir=kind, potential=potential,
                 pump_terms=lasers)
    eng.set_pump(env.astype(eng.real) if lasers > 1 else env[0].astype(eng.real))
    if potential:
        eng.set_potential(pot.astype(eng.real))
    if noise:
        eng.set_noise([31], P["gamma_C"], P["R"], 1.0, dt / (4 * dx * dy))
    res = None if not fields else fields[0] if len(fields) == 1 else np.stack(fields)
    eng.set_state(psi0.astype(eng.complex), None if res is None else res.astype(eng.real))
    scales = np.array([[[coeff(l, (k + f) * dt) for l in range(lasers)] for f in (0.25, 0.75)] for k in range(steps)])
    eng.split_advance(0 if ordering == "cpu" else 1, 0, steps,
                      scales.reshape((steps, 2) + ((lasers,) if lasers > 1 else ()) + (1,)))
    psi, res = eng.get_state()
    eng.close()
    if ordering == "kouter":
        psi = np.fft.ifft2(psi.astype(np.complex128), axes=(-2, -1))
    k2 = np.add.outer((2 * np.pi * np.fft.fftfreq(ny, d=dy)) ** 2, (2 * np.pi * np.fft.fftfreq(nx, d=dx)) ** 2)
    draw = gpe.Noise([31], [P["gamma_C"]], [P["R"]], [1.0], dt, dx * dy, "double",
                     normals_precision="single") if noise else None
    want, want_f = gpe.split_advance(ordering, psi0.copy(), tuple(f.copy() for f in fields),
                                     lambda t: sum(env[l] * coeff(l, t) for l in range(lasers)), pot, P, k2, dx, dy,
                                     dt, 0, steps, kind=kind, noise=draw)
    assert rel_l2(psi, want) < 1.5e-5
    for q, f in enumerate(want_f):
        assert rel_l2(res if len(want_f) == 1 else res[q], f) < 1.5e-5, q
