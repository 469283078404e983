"""Rounding of the FP64 split-step kick.

A plane wave on a 4 x 4 grid without potential, interaction, gain or pump: its transforms are sums of
equal terms times +-1 and +-i, exact in binary, so a step's only rounding is that of its two kinetic
half kicks on the one mode that is not zero.  A kick that rounds psi once leaves an error of the
rounding of its two components, 4.7e-17 of |psi| rms over the mantissa's range, and N independent
ones sqrt(N) times that; one that rounds twice sqrt(2) times more.  256 amplitudes give the rms to
some 5 %, so the line lies at 1.2."""
from __future__ import annotations

import math

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_fp64_kick_rounds_psi_once(cuda_lib):
    from polarism_gb300.engine import Engine, MemberPhysics

    members, steps, n, dx, dy, dt = 256, 512, 4, 8.0, 7.0, 0.02
    p = MemberPhysics(g_C=0.0, g_R=0.0, R=0.0, gamma_C=0.0, gamma_R=0.0)
    rng = np.random.default_rng(2)
    amp = rng.uniform(1.0, 2.0, members) * np.exp(2j * np.pi * rng.random(members))
    wave = np.array([1, 1j, -1, -1j])
    psi0 = amp[:, None, None, None] * (wave[None, :] * wave[:, None])[None, None]
    eng = Engine(n, n, members, dx, dy, dt, p, "double")
    eng.set_pump(np.zeros((n, n)))
    eng.set_state(psi0, np.zeros((members, 1, n, n)))
    eng.split_advance(0, 0, steps, np.zeros((steps, 2, members)))
    psi, _ = eng.get_state()
    eng.close()
    L = np.longdouble
    factor = (L(1), L(0))
    for d in (dx, dy):
        k = 2 * math.pi / (n * d)
        theta = p.hbar * 0.5 * dt / (2 * p.m_eff) * k * k
        sh = math.sin(0.5 * theta)
        re, im = 1 + L(-2 * sh * sh), L(-math.sin(theta))
        factor = (factor[0] * re - factor[1] * im, factor[0] * im + factor[1] * re)
    want = (amp.real.astype(L), amp.imag.astype(L))
    for _ in range(2 * steps):
        want = (want[0] * factor[0] - want[1] * factor[1], want[0] * factor[1] + want[1] * factor[0])
    got = psi[:, 0, 0, 0]
    err = np.hypot(got.real.astype(L) - want[0], got.imag.astype(L) - want[1]) / np.abs(amp)
    assert float(np.sqrt(np.mean(err ** 2))) < 1.2 * 4.7e-17 * math.sqrt(2 * steps)
