"""FP32 IFRK passes on the register-resident transforms, one and two components, every size along
both axes and every kind of site step, against the FP64 oracle.

Tolerance of the fields: a step makes at most seven stages of four one-axis transforms of at most
log2(4096) = 12 rounded levels, each stage's result scaled by the step into psi, and psi itself passes
through one chain of them; three steps are some 1000 roundings of 6e-8, 2e-6 as a random walk and
6e-5 adding up at worst.  The error norm is a root mean square of sums of a few stage spectra that carry
a relative rounding of about 1e-6 each against a scale of 1e-4 of psi: 1e-3 of an estimate that is
well above one."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import gpe
from tests.conftest import rel_l2

pytestmark = pytest.mark.gpu

P = dict(hbar=0.6582119514, m_eff=0.284, g_C=0.02, g_R=0.03, g_I=0.01, R=0.05, gamma_C=0.083, gamma_R=0.02,
         gamma_I=0.01, gamma_A=0.03, R_IA=0.05, R_AI=0.01, kappa=0.05, kinetic_relaxation_eta=0.0)
SPIN = dict(alpha_2=-0.004, zeeman=0.05, te_tm=0.03)
WEIGHTS = (0.7, 0.3)
SIZES = [(64, 64), (64, 128), (128, 64), (256, 8), (8, 256), (512, 4), (4, 512), (1024, 16), (16, 1024),
         (2048, 8), (8, 2048), (4096, 4), (4, 4096)]


class Case:
    """A field with every term the configuration has, and its oracle."""

    def __init__(self, ny, nx, kind="single", components=1, res_components=None, lasers=1, potential=0, seed=1):
        self.nx, self.ny, self.kind, self.comps, self.lasers, self.potential = nx, ny, kind, components, lasers, potential
        self.rc = res_components or components
        self.dx, self.dy, self.dt = 1.1, 0.9, 0.02
        rng = np.random.default_rng(seed + 7 * nx + 11 * ny)
        self.psi0 = 0.5 * (rng.standard_normal((1, components, ny, nx))
                           + 1j * rng.standard_normal((1, components, ny, nx)))
        fields = {"none": 0, "single": 1, "double": 2, "quadratic-double": 2}[kind]
        self.res0 = tuple(rng.random((1, self.rc, ny, nx)) for _ in range(fields))
        self.env = rng.random((lasers, ny, nx))
        pot = 0.05 * rng.standard_normal((ny, nx))
        self.pot = (0.0, pot, pot - 0.01j * rng.random((ny, nx)))[potential]
        self.kx, self.ky = np.meshgrid(2 * np.pi * np.fft.fftfreq(nx, d=self.dx),
                                       2 * np.pi * np.fft.fftfreq(ny, d=self.dy), indexing="xy")
        self.p = dict(P, **(SPIN if components == 2 else {}))
        self.spin = dict(kx=self.kx, ky=self.ky, weights=np.array([WEIGHTS])) if components == 2 else None

    def coeff(self, l, t):
        return 0.3 * (1.0 + 0.2 * l) * (1.0 + 0.4 * np.sin(9 * t + l))

    def pump(self, t):
        return sum(self.env[l] * self.coeff(l, t) for l in range(self.lasers))

    def engine(self, precision="single", noise=False):
        from polarism_gb300.engine import Engine, MemberPhysics

        phys = MemberPhysics(**self.p, **(dict(pump_weight_plus=WEIGHTS[0], pump_weight_minus=WEIGHTS[1])
                                          if self.comps == 2 else {}))
        eng = Engine(self.nx, self.ny, 1, self.dx, self.dy, self.dt, phys, precision, reservoir=self.kind,
                     potential=self.potential, components=self.comps, reservoir_components=self.rc,
                     pump_terms=self.lasers)
        eng.set_pump(self.env.astype(eng.real) if self.lasers > 1 else self.env[0].astype(eng.real))
        if self.potential:
            eng.set_potential(self.pot.astype(eng.complex if self.potential == 2 else eng.real))
        if noise:
            eng.set_noise([9], self.p["gamma_C"], self.p["R"], 1.0, self.dt / (4 * self.dx * self.dy))
        res = None
        if self.res0:
            res = self.res0[0] if len(self.res0) == 1 else np.stack(self.res0)
        eng.set_state(self.psi0.astype(eng.complex),
                      None if res is None else np.ascontiguousarray(res, dtype=eng.real))
        return eng

    def scales(self, tableau, steps):
        from polarism_gb300.engine import TABLEAU_NODES

        rows = [[[self.coeff(l, (k + c) * self.dt) for l in range(self.lasers)] for c in TABLEAU_NODES[tableau]]
                for k in range(steps)]
        return np.asarray(rows).reshape((steps, -1) + ((self.lasers,) if self.lasers > 1 else ()) + (1,))

    def step(self, state, h, tableau, **kw):
        return gpe.ifrk_step(state, h, gpe.TABLEAUS[tableau], self.pump, self.pot, self.p,
                             self.kx ** 2 + self.ky ** 2, self.dx, self.dy, kind=self.kind, spinor=self.spin, **kw)


@pytest.mark.parametrize("ny,nx", SIZES)
@pytest.mark.parametrize("tableau,noise,config", [
    ("rk4", True, dict()),
    ("dp5", False, dict(potential=2)),
    ("rk4", False, dict(kind="none", potential=1)),
    ("rk4", True, dict(kind="quadratic-double", lasers=2)),
    ("rk4", True, dict(kind="double", components=2)),
    ("dp5", False, dict(kind="single", components=2, res_components=1, potential=1)),
    ("rk4", False, dict(kind="double", components=2, res_components=1, lasers=2)),
    ("rk4", True, dict(kind="single", components=2))],
    ids=["noise", "dp5-complex", "no-reservoir", "quadratic-double-lasers", "spinor-double-noise",
         "spinor-shared-dp5", "spinor-shared-double-lasers", "spinor-noise"])
def test_fixed_steps_match_oracle(cuda_lib, ny, nx, tableau, noise, config):
    c = Case(ny, nx, **config)
    steps = 3
    eng = c.engine(noise=noise)
    eng.ifrk_advance(tableau, 0, steps, c.scales(tableau, steps))
    psi, res = eng.get_state()
    eng.close()
    draw = gpe.Noise([9], [c.p["gamma_C"]], [c.p["R"]], [1.0], c.dt, c.dx * c.dy, "double",
                     normals_precision="single")
    state = gpe.IFRKState(psi=c.psi0.copy(), fields=tuple(r.copy() for r in c.res0))
    for k in range(steps):
        c.step(state, c.dt, tableau)
        state.psi, state.psi_k = state.real_space(), None
        if noise:
            draw.apply(state.psi, state.fields[0], k)
    assert rel_l2(psi, state.psi) < 6e-5
    for q, want in enumerate(state.fields):
        got = res if len(state.fields) == 1 else res[q]
        assert rel_l2(got, want) < 6e-5, q


@pytest.mark.parametrize("ny,nx", SIZES)
@pytest.mark.parametrize("config", [dict(), dict(kind="double", components=2)], ids=["scalar", "spinor"])
def test_error_norm_matches_oracle(cuda_lib, ny, nx, config):
    c = Case(ny, nx, **config)
    c.dt, h = 1e-3, 0.6  # pump coefficients of a trial are given at its own nodes
    eng = c.engine()
    from polarism_gb300.engine import TABLEAU_NODES

    scales = np.asarray([[c.coeff(0, node * h)] for node in TABLEAU_NODES["dp5"]])
    err, accepted = eng.ifrk_trial(h, scales, 1e-4, 1e-6)
    eng.close()
    state = gpe.IFRKState(psi=c.psi0.copy(), fields=c.res0)
    want = c.step(state, h, "dp5", adaptive=True, rtol=1e-4, atol=1e-6)
    assert want > 1.2  # far above what FP32 adds
    assert abs(err - want) <= 1e-3 * want and not accepted
