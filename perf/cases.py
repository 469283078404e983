"""Workloads of the time-stepping framework that its speed is measured on.

Each case is what a user has the framework do between two looks at the state: a chunk of steps
of one solver (fused RK4, split-step Fourier in both orderings, Lawson IFRK, the uneven sweep),
or one training step of the warm-start network.  Sizes are those of the framework's own
configurations (128^2, 256^2, 512^2, 1024^2, 4096^2 grids, one to tens of members) and ragged
ones between them.

``listed()`` names the cases, ``draw(rng)`` gives more of the same ranges, ``prepare(case,
seed)`` makes inputs and the solver handle, ``run(state)`` is one pass through the public entry
points, ``work(case)`` counts its unavoidable bytes and flops and ``exact(case, seed)`` is the
same pass in 64 bits in plain torch.
"""
from __future__ import annotations

import math

import numpy as np
import torch

HBAR = 0.6582119514
PHYSICS = dict(hbar=HBAR, m_eff=0.284, g_C=0.001, g_R=0.002, g_I=0.0, R=0.02, gamma_C=0.083,
               gamma_R=0.005)
SPINOR = dict(PHYSICS, g_I=0.0005, alpha_2=-1e-4, zeeman=0.05, te_tm=0.05, gamma_I=0.001,
              gamma_A=0.005, R_IA=0.05, R_AI=0.0025, pump_weight_plus=0.5, pump_weight_minus=0.5)
DOUBLE = dict(PHYSICS, g_I=0.0005, gamma_I=0.001, gamma_A=0.005, R_IA=0.05, R_AI=0.0025)


def _grid_case(name, kind, nx, ny, members, steps, **options):
    """One grid solver's chunk: ``precision``, ``noise`` (truncated Wigner), ``potential`` (none,
    real, complex), ``reservoir`` (single, double), ``spacing`` (um) and ``dt`` (ps)."""
    case = dict(name=name, kind=kind, nx=nx, ny=ny, members=members, steps=steps, precision="single",
                noise=True, potential="none", reservoir="single", spacing=0.390625, dt=5e-4)
    case.update(options)
    return case if name else {key: value for key, value in case.items() if key != "name"}


def listed():
    return [
        # The smallest call: the plain-method configuration (128^2, double, dt 1e-3), one short
        # chunk of a single simulation; nothing but latency and launches.
        _grid_case("rk4-128-double", "rk4", 128, 128, 1, 16, precision="double", noise=False,
                   spacing=0.78125, dt=1e-3),
        # The solver class as the simulation controller calls it, on host arrays: the default
        # 256^2 grid in single precision with Wigner noise, one sampling interval.
        _grid_case("dropin-256-host", "dropin", 256, 256, 1, 200, dt=1e-3),
        # A sample that is no power of two, with a disorder potential and a few seeds.
        _grid_case("rk4-600x500-potential", "rk4", 600, 500, 6, 64, potential="real", spacing=0.2),
        # The headline: 1024^2 with Wigner noise, several noise trajectories together.
        _grid_case("rk4-1024x8", "rk4", 1024, 1024, 8, 64),
        # The largest single field: one 4096^2 sample.
        _grid_case("rk4-4096", "rk4", 4096, 4096, 1, 16),
        # A parameter sweep over mixed grids (128^2, 256^2, 512^2, a third each), no noise.
        dict(name="sweep-48-mixed", kind="sweep", small=16, middle=16, large=16, steps=64, noise=False,
             dt=1e-3),
        # The same physics stepped spectrally, the spectrum kept between steps.
        _grid_case("split-kouter-1024x8", "split1", 1024, 1024, 8, 32),
        # Spectral steps in the CPU solver's order on a middle grid, a few members.
        _grid_case("split-512x4", "split0", 512, 512, 4, 32),
        # One double-precision spectral run, as the precision check makes them.
        _grid_case("split-256-double", "split0", 256, 256, 1, 16, precision="double"),
        # Lawson integrating-factor RK4 at fixed steps on a middle grid.
        _grid_case("ifrk4-512x4", "ifrk4", 512, 512, 4, 16, dt=5e-3),
        # The spinor configuration: two components, TE-TM and Zeeman splitting, double reservoir,
        # ring pump, adaptive Dormand-Prince trials.
        dict(name="spinor-dp5-512", kind="dp5", nx=512, ny=512, steps=4, h=0.2, spacing=0.25),
        # One optimiser step of the warm-start network on a batch of pumps at its full grid.
        dict(name="fno-train-256x8", kind="fno", n=256, batch=8, width=32, modes=16, layers=4,
             hidden=128),
    ]


def _log_int(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def _steps_for(sites, budget, low=4, high=128):
    return max(low, min(high, budget // max(1, sites)))


def draw(rng):
    kind = rng.choice(["rk4", "rk4", "rk4", "dropin", "sweep", "split0", "split1", "ifrk4", "dp5", "fno"])
    if kind in ("rk4", "dropin"):
        shape = rng.choice(["power", "ragged", "wide"])
        if shape == "power":
            nx = ny = 2 ** rng.randint(6, 11)
        elif shape == "ragged":
            nx, ny = _log_int(rng, 60, 1500), _log_int(rng, 60, 1500)
        else:
            nx, ny = 1024 * rng.randint(1, 4), _log_int(rng, 64, 2048)
        double = kind == "rk4" and rng.random() < 0.25
        most = (2 ** 19 if double else 2 ** 23) if kind == "rk4" else 2 ** 18
        members = max(1, min(8, _log_int(rng, 1, 8), most // (nx * ny)))
        if double:
            while nx * ny > most:
                nx, ny = max(4, nx // 2), max(4, ny // 2)
        steps = _steps_for(nx * ny * members, 2 ** 22 if double else 2 ** 27)
        return _grid_case(None, kind, nx, ny, members, steps, precision="double" if double else "single",
                          noise=rng.random() < 0.7,
                          potential=rng.choice(["none", "none", "real", "complex"]) if kind == "rk4" else "none",
                          reservoir=rng.choice(["single", "single", "single", "double"]) if kind == "rk4" else "single",
                          spacing=rng.choice([0.25, 0.390625, 0.5]), dt=rng.choice([2.5e-4, 5e-4]))
    if kind == "sweep":
        return dict(kind="sweep", small=rng.randint(1, 16), middle=rng.randint(1, 16),
                    large=rng.randint(1, 16), steps=rng.choice([32, 48, 64]), noise=rng.random() < 0.5, dt=1e-3)
    if kind in ("split0", "split1", "ifrk4"):
        nx, ny = 2 ** rng.randint(6, 11), 2 ** rng.randint(6, 11)
        double = kind != "ifrk4" and rng.random() < 0.25
        most = 2 ** 18 if double else 2 ** 22
        while nx * ny > most:
            nx, ny = nx // 2, ny // 2
        members = max(1, min(8, _log_int(rng, 1, 8), most // (nx * ny)))
        budget = 2 ** 20 if double else (2 ** 25 if kind != "ifrk4" else 2 ** 23)
        steps = _steps_for(nx * ny * members, budget, high=64)
        return _grid_case(None, kind, nx, ny, members, steps, precision="double" if double else "single",
                          noise=rng.random() < 0.7,
                          potential=rng.choice(["none", "none", "real", "complex"]),
                          reservoir=rng.choice(["single", "single", "single", "double"]),
                          spacing=rng.choice([0.25, 0.390625, 0.5]),
                          dt=rng.choice([2.5e-4, 5e-4]) if kind != "ifrk4" else rng.choice([2e-3, 5e-3]))
    if kind == "dp5":
        n = 2 ** rng.randint(6, 9)
        return dict(kind="dp5", nx=n, ny=2 ** rng.randint(6, 9), steps=rng.randint(2, 4),
                    h=rng.choice([0.1, 0.15, 0.2]), spacing=rng.choice([0.25, 0.5]))
    return dict(kind="fno", n=rng.choice([64, 96, 128, 200, 256]), batch=rng.randint(1, 8), width=32,
                modes=rng.choice([12, 16]), layers=4, hidden=128)


# ------------------------------------------------------------------------------- inputs
def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _generator(seed, stream):
    g = torch.Generator(device=_device())
    g.manual_seed((int(seed) * 1_000_003 + 7919 * stream + 17) % (2 ** 62))
    return g


def _radius2(nx, ny, spacing):
    x = (torch.arange(nx, dtype=torch.float64, device=_device()) - (nx - 1) / 2) * spacing
    y = (torch.arange(ny, dtype=torch.float64, device=_device()) - (ny - 1) / 2) * spacing
    return x, y, x[None, :] ** 2 + y[:, None] ** 2


def _smooth(nx, ny, g):
    """A smooth order-one random landscape: a few plane waves of random phase."""
    x = torch.arange(nx, dtype=torch.float64, device=_device()) * (2 * math.pi / nx)
    y = torch.arange(ny, dtype=torch.float64, device=_device()) * (2 * math.pi / ny)
    out = torch.zeros((ny, nx), dtype=torch.float64, device=_device())
    phases = torch.rand((6,), generator=g, device=_device(), dtype=torch.float64) * (2 * math.pi)
    for (a, b), p in zip(((1, 0), (0, 1), (1, 2), (2, -1), (3, 1), (-2, 3)), phases):
        out = out + torch.cos(a * x[None, :] + b * y[:, None] + p)
    return out / 6


def _real(case):
    return torch.float64 if case.get("precision") == "double" else torch.float32


def _complex(case):
    return torch.complex128 if case.get("precision") == "double" else torch.complex64


def _inputs(case, seed):
    """Fields of a running simulation: a Gaussian (or ring) condensate with noise on it above a
    partly filled reservoir, the pump envelope, a disorder potential."""
    nx, ny, spacing = case["nx"], case["ny"], case["spacing"]
    members = case.get("members", 1)
    comps = 2 if case["kind"] == "dp5" else 1
    g = _generator(seed, 1)
    rt, ct = _real(case), _complex(case)
    _, _, r2 = _radius2(nx, ny, spacing)
    size = spacing * min(nx, ny)
    envs, psis = [], []
    for m in range(members):
        u = float(torch.rand((1,), generator=g, device=_device()))
        if case["kind"] == "dp5":
            env = torch.exp(-0.5 * ((torch.sqrt(r2) - 0.23 * size) / (0.03 * size)) ** 2)
        else:
            env = torch.exp(-0.5 * r2 / ((0.08 + 0.1 * u) * size) ** 2)
        envs.append(env.to(rt))
        per_comp = []
        for c in range(comps):
            noise = torch.randn((ny, nx, 2), generator=g, device=_device(), dtype=torch.float64)
            phase = _smooth(nx, ny, g) * 2.0
            body = 0.6 * env.sqrt() * (1.0 - 0.3 * c)
            per_comp.append(torch.complex(body * torch.cos(phase) + 0.03 * noise[..., 0],
                                          body * torch.sin(phase) + 0.03 * noise[..., 1]).to(ct))
        psis.append(torch.stack(per_comp))
    psi = torch.stack(psis).contiguous()
    env = torch.stack(envs)[:, None].contiguous()
    fields = 2 if case.get("reservoir") == "double" or case["kind"] == "dp5" else 1
    n = []
    for f in range(fields):
        bump = torch.rand((members, comps, ny, nx), generator=g, device=_device(), dtype=torch.float64)
        n.append(((3.5 - 1.5 * f) * env.double() * (0.9 + 0.2 * bump) + 0.01 * bump).to(rt))
    res = n[0].contiguous() if fields == 1 else torch.stack(n).contiguous()
    pot = None
    if case.get("potential", "none") != "none":
        v = _smooth(nx, ny, g) * 0.5
        pot = v.to(rt) if case["potential"] == "real" else torch.complex(v, -0.05 * _smooth(nx, ny, g) ** 2).to(ct)
        pot = pot.contiguous()
    seeds = [int(seed) * 64 + 42 + m for m in range(members)]
    return dict(psi=psi, res=res, env=env, pot=pot, seeds=seeds)


P0 = 0.4


def _physics(case):
    return SPINOR if case["kind"] == "dp5" else DOUBLE if case.get("reservoir") == "double" else PHYSICS


def _grid_engine(case, x):
    from polarism_gb300.engine import Engine, MemberPhysics

    spinor = case["kind"] == "dp5"
    members = case.get("members", 1)
    eng = Engine(case["nx"], case["ny"], members, case["spacing"], case["spacing"],
                 case["h"] if spinor else case["dt"], MemberPhysics(**_physics(case)),
                 case.get("precision", "single"), reservoir="double" if spinor else case["reservoir"],
                 potential={"none": 0, "real": 1, "complex": 2}[case.get("potential", "none")],
                 pump_per_member=members > 1, components=2 if spinor else 1)
    eng.set_pump(x["env"])
    if x["pot"] is not None:
        eng.set_potential(x["pot"])
    if case.get("noise"):
        eng.set_noise(x["seeds"], PHYSICS["gamma_C"], PHYSICS["R"], 1.0,
                      case["dt"] / (4 * case["spacing"] ** 2))
    return eng


SWEEP_SIZES = (("small", 128), ("middle", 256), ("large", 512))


def _sweep_inputs(case, seed):
    """Members in random order of size, each packed after the one before."""
    sizes = [n for key, n in SWEEP_SIZES for _ in range(case[key])]
    order = torch.randperm(len(sizes), generator=_generator(seed, 2), device=_device()).tolist()
    sizes = [sizes[i] for i in order]
    parts = []
    for m, n in enumerate(sizes):
        one = dict(kind="rk4", nx=n, ny=n, members=1, spacing=0.5, reservoir="single")
        parts.append(_inputs(one, int(seed) * 977 + m))
    return dict(sizes=sizes, psi=torch.cat([p["psi"].reshape(-1) for p in parts]),
                res=torch.cat([p["res"].reshape(-1) for p in parts]),
                envs=[p["env"][0, 0] for p in parts], seeds=[int(seed) * 512 + m for m in range(len(sizes))])


def _fno_params(case, seed):
    rng = np.random.default_rng(int(seed) + 11)
    w, m, h = case["width"], case["modes"], case["hidden"]
    p = {"lift_w": rng.standard_normal((w, 3)) / math.sqrt(3), "lift_b": 0.1 * rng.standard_normal(w)}
    for k in range(case["layers"]):
        p[f"spec{k}_re"] = rng.uniform(-1, 1, (2 * m, m, w, w)) / (w * w)
        p[f"spec{k}_im"] = rng.uniform(-1, 1, (2 * m, m, w, w)) / (w * w)
        p[f"w{k}"] = rng.standard_normal((w, w)) / math.sqrt(w)
        p[f"b{k}"] = 0.1 * rng.standard_normal(w)
    p["proj1_w"] = rng.standard_normal((h, w)) / math.sqrt(w)
    p["proj1_b"] = 0.1 * rng.standard_normal(h)
    p["proj2_w"] = rng.standard_normal((3, h)) / math.sqrt(h)
    p["proj2_b"] = 0.1 * rng.standard_normal(3)
    return p


def _fno_inputs(case, seed):
    """Pumps in threshold units with the coordinates, and steady-state-like targets."""
    n, batch = case["n"], case["batch"]
    g = _generator(seed, 3)
    x, y, r2 = _radius2(n, n, 128.0 / n)
    feats, targets = [], []
    for _ in range(batch):
        u = torch.rand((2,), generator=g, device=_device(), dtype=torch.float64)
        env = torch.exp(-0.5 * r2 / (8.0 + 12.0 * u[0]) ** 2)
        feats.append(torch.stack([env * (1.0 + 2.0 * u[1]), (x / 64.0)[None, :].expand(n, n),
                                  (y / 64.0)[:, None].expand(n, n)]))
        phase = r2 / 900.0
        targets.append(torch.stack([env * torch.cos(phase), env * torch.sin(phase), 4.0 * env / (1 + env)]))
    return (torch.stack(feats).float().contiguous(), torch.stack(targets).float().contiguous())


# ------------------------------------------------------------------------------- the pass
SAMPLES = {"rk4": 3, "split0": 2, "split1": 2, "ifrk4": 4, "dp5": 7}


def prepare(case, seed):
    kind = case["kind"]
    if kind == "fno":
        from polarism_gb300.fno import FNO2d

        a, target = _fno_inputs(case, seed)
        net = FNO2d(case["n"], width=case["width"], modes=case["modes"], layers=case["layers"],
                    hidden=case["hidden"], params=_fno_params(case, seed))
        torch.cuda.synchronize()
        return dict(case=case, net=net, a=a, target=target)
    if kind == "sweep":
        from polarism_gb300.engine import MemberPhysics
        from polarism_gb300.sweep import SweepEngine, autotune_tiling

        x = _sweep_inputs(case, seed)
        members = len(x["sizes"])
        eng = SweepEngine([(n, n, 0.5, 0.5) for n in x["sizes"]], [MemberPhysics(**PHYSICS)] * members,
                          case["dt"])
        eng.set_pump([e.cpu().numpy() for e in x["envs"]])
        if case["noise"]:
            ones = np.ones(members)
            eng.set_noise(x["seeds"], PHYSICS["gamma_C"] * ones, PHYSICS["R"] * ones, ones)
        torch.cuda.synchronize()
        autotune_tiling(eng, noise=case["noise"], use_cache=False)  # as a sweep run does before its steps
        return dict(case=case, eng=eng, psi=x["psi"], res=x["res"], psi_out=torch.empty_like(x["psi"]),
                    res_out=torch.empty_like(x["res"]), scales=np.full((case["steps"], 3, members), P0))
    if kind == "dropin":
        return _prepare_dropin(case, seed)
    x = _inputs(case, seed)
    torch.cuda.synchronize()  # the handle copies device arrays on its own stream
    eng = _grid_engine(case, x)
    members = case.get("members", 1)
    lead = (SAMPLES[kind],) if kind == "dp5" else (case["steps"], SAMPLES[kind])
    return dict(case=case, eng=eng, psi=x["psi"], res=x["res"], psi_out=torch.empty_like(x["psi"]),
                res_out=torch.empty_like(x["res"]), scales=np.full(lead + (members,), P0))


def _prepare_dropin(case, seed):
    from polarism_gb300 import host
    from polarism_gb300.solvers import RK4CudaSolver

    cfg = host.Config()
    cfg.grid.nx, cfg.grid.ny = case["nx"], case["ny"]
    cfg.grid.lx, cfg.grid.ly = case["nx"] * case["spacing"], case["ny"] * case["spacing"]
    cfg.solver.precision, cfg.solver.dt = case["precision"], case["dt"]
    cfg.laser.P0, cfg.laser.sigma_space = P0, 0.12 * case["spacing"] * min(case["nx"], case["ny"])
    cfg.noise.stochastic = "wigner" if case["noise"] else "none"
    configs = []
    for m in range(case["members"]):
        c = host.copy_config(cfg)
        c.noise.seed = int(seed) * 64 + 42 + m
        configs.append(c)
    grid, model, state = host.build_simulation(configs[0], configs if case["members"] > 1 else None)
    x = _inputs(case, seed)
    psi, res = x["psi"].cpu().numpy(), x["res"].cpu().numpy()
    state.field = psi.copy()
    model.reservoir.set_state((res.copy(),))
    solver = RK4CudaSolver(configs[0], grid, model)
    return dict(case=case, solver=solver, model=model, state=state)


def run(state):
    case = state["case"]
    kind, steps = case["kind"], case.get("steps", 1)
    if kind == "fno":
        net = state["net"]
        out, cache = net.forward(state["a"])
        loss, grad = net.mse(out, state["target"])
        grads = net.backward(cache, grad)
        net.adam_step(grads)
        return {"out": out, "loss": loss, "grads": grads}
    if kind == "dropin":
        state["solver"].advance(state["model"], state["state"], steps)
        return {"psi": state["state"].field, "res": state["model"].reservoir.get_state()[0]}
    eng, psi, res = state["eng"], state["psi_out"], state["res_out"]
    eng.set_state(state["psi"], state["res"])
    if kind == "sweep":
        from polarism_gb300 import _lib

        eng.advance(0, steps, state["scales"])
        _lib.check(_lib.load().pg_sweep_get_state(eng._h, psi.data_ptr(), res.data_ptr(), 1), "pg_sweep_get_state")
        return {"psi": psi, "res": res}
    if kind == "dp5":
        for _ in range(steps):
            eng.ifrk_trial(case["h"], state["scales"], 1e-3, 1e-5)
    else:
        eng.set_state_kind(False)
        if kind == "rk4":
            eng.advance(0, steps, state["scales"])
        elif kind == "ifrk4":
            eng.ifrk_advance("rk4", 0, steps, state["scales"])
        else:
            eng.split_advance(1 if kind == "split1" else 0, 0, steps, state["scales"])
    eng.get_state(psi, res)
    return {"psi": psi, "res": res}


# ------------------------------------------------------------------------------- work
def work(case):
    """Bytes: each step reads and writes the field and the reservoir and reads the pump once; a
    2-D transform takes two passes over the field."""
    kind = case["kind"]
    if kind == "fno":
        n, b, w, m, h = case["n"], case["batch"], case["width"], case["modes"], case["hidden"]
        sites = float(b * n * n)
        dft = 2 * sites * w * 2 * m + 8.0 * b * w * n * m * 2 * m
        mixing = 8.0 * b * w * w * 2 * m * m
        layer = 2 * dft + mixing + 2 * sites * w * w
        forward = 2 * sites * (3 * w + w * h + 3 * h) + case["layers"] * layer
        weights = case["layers"] * (4.0 * m * m * w * w + w * w) + w * h
        return {"bytes": 4 * sites * 9 + 2 * sites * w * (case["layers"] + 1) * 2 + 28 * weights,
                "flops": 3 * forward}
    if kind == "sweep":
        sites = sum(case[key] * n * n for key, n in SWEEP_SIZES)
        return {"bytes": 28.0 * sites * case["steps"], "flops": (260.0 if case["noise"] else 200.0) * sites * case["steps"]}
    real = 8 if case.get("precision") == "double" else 4
    sites = float(case["nx"] * case["ny"] * case.get("members", 1)) * case["steps"]
    fields = 2 if case.get("reservoir") == "double" or kind == "dp5" else 1
    pot = {"none": 0, "real": 1, "complex": 2}[case.get("potential", "none")]
    local = 2 * fields + 1 + pot
    butterflies = 5.0 * math.log2(case["nx"] * case["ny"])
    extra = 60.0 if case.get("noise") else 0.0
    if kind in ("rk4", "dropin"):
        return {"bytes": real * sites * (4 + local), "flops": sites * (200 + extra)}
    if kind == "split1":
        return {"bytes": real * sites * (8 + local), "flops": sites * (2 * butterflies + 70 + extra)}
    if kind == "split0":
        return {"bytes": real * sites * (16 + local), "flops": sites * (4 * butterflies + 90 + extra)}
    stages, comps = (5, 1) if kind == "ifrk4" else (9, 2)
    return {"bytes": real * sites * comps * stages * (8 + local - fields),
            "flops": sites * comps * stages * (2 * butterflies + 60)}


# ------------------------------------------------------------------------------- 64 bits
def _philox(cell, step, key):
    """Philox-4x32-10 words of the counters (cell, step low, step high, 1) as int64 tensors."""
    mask = 0xFFFFFFFF
    a, b, c, d = cell, torch.full_like(cell, step & mask), torch.full_like(cell, step >> 32), torch.ones_like(cell)
    k0, k1 = key & mask, key >> 32

    def wide(v, multiplier):
        low = v * (multiplier & 0xFFFF)
        high = v * (multiplier >> 16) + (low >> 16)
        return high >> 16, ((high & 0xFFFF) << 16) | (low & 0xFFFF)

    for _ in range(10):
        h0, l0 = wide(a, 0xD2511F53)
        h1, l1 = wide(c, 0xCD9E8D57)
        a, b, c, d = h1 ^ b ^ k0, l1, h0 ^ d ^ k1, l0
        k0, k1 = (k0 + 0x9E3779B9) & mask, (k1 + 0xBB67AE85) & mask
    return a, b, c, d


def _normals(nx, ny, step, key, double):
    cell = torch.arange(nx * ny, dtype=torch.int64, device=_device()).reshape(ny, nx)
    a, b, c, d = _philox(cell, step, key)
    if double:
        u1 = ((a >> 5).double() * 67108864.0 + (b >> 6).double() + 1.0) * 2.0 ** -53
        u2 = ((c >> 5).double() * 67108864.0 + (d >> 6).double() + 1.0) * 2.0 ** -53
    else:
        u1, u2 = ((a >> 8) + 1).double() * 2.0 ** -24, ((b >> 8) + 1).double() * 2.0 ** -24
    r = torch.sqrt(-2.0 * torch.log(u1))
    return torch.polar(r, 2 * math.pi * u2)


def _wigner(psi, n_active, step, seeds, p, dt, cell, double):
    out = psi.clone()
    ny, nx = psi.shape[-2:]
    for m, key in enumerate(seeds):
        var = (p["gamma_C"] + p["R"] * n_active[m, 0]) * dt / (4 * cell)
        out[m, 0] += torch.sqrt(var) * _normals(nx, ny, step, key, double)
    return out


def _res_rates(fields, rho, pump, p):
    if len(fields) == 1:
        return [pump - (p["gamma_R"] + p["R"] * rho) * fields[0]]
    a, i = fields
    return [p["R_IA"] * i - (p["gamma_A"] + p["R_AI"] + p["R"] * rho) * a,
            pump - (p["gamma_I"] + p["R_IA"]) * i + p["R_AI"] * a]


def _potential_energy(fields, p):
    return p["g_R"] * fields[0] + (p["g_I"] * fields[1] if len(fields) == 2 else 0.0)


def _density(psi):
    return psi.real ** 2 + psi.imag ** 2


def _rk4_exact(psi, fields, pump, pot, p, spacing, dt, steps, seeds, double):
    kin = p["hbar"] / (2 * p["m_eff"]) / spacing ** 2

    def rhs(y, f):
        rho = _density(y)
        lap = torch.roll(y, 1, -1) + torch.roll(y, -1, -1) + torch.roll(y, 1, -2) + torch.roll(y, -1, -2) - 4 * y
        energy = p["g_C"] * rho + _potential_energy(f, p) + pot
        gain = 0.5 * (p["R"] * f[0] - p["gamma_C"])
        return 1j * kin * lap + (gain - 1j / p["hbar"] * energy) * y, _res_rates(f, rho, pump, p)

    for k in range(steps):
        k1, r1 = rhs(psi, fields)
        k2, r2 = rhs(psi + 0.5 * dt * k1, [n + 0.5 * dt * r for n, r in zip(fields, r1)])
        k3, r3 = rhs(psi + 0.5 * dt * k2, [n + 0.5 * dt * r for n, r in zip(fields, r2)])
        k4, r4 = rhs(psi + dt * k3, [n + dt * r for n, r in zip(fields, r3)])
        psi = psi + dt / 6 * (k1 + 2 * k2 + 2 * k3 + k4)
        fields = [(n + dt / 6 * (a + 2 * b + 2 * c + d)).clamp_min(0)
                  for n, a, b, c, d in zip(fields, r1, r2, r3, r4)]
        if seeds is not None:
            psi = _wigner(psi, fields[0], k, seeds, p, dt, spacing ** 2, double)
    return psi, fields


def _k_axes(nx, ny, spacing):
    kx = 2 * math.pi * torch.fft.fftfreq(nx, d=spacing, dtype=torch.float64, device=_device())
    ky = 2 * math.pi * torch.fft.fftfreq(ny, d=spacing, dtype=torch.float64, device=_device())
    return kx[None, :], ky[:, None]


def _split_exact(psi, fields, pump, pot, p, spacing, dt, steps, seeds, double, kouter):
    kx, ky = _k_axes(psi.shape[-1], psi.shape[-2], spacing)
    theta = p["hbar"] * dt * (kx ** 2 + ky ** 2) / (2 * p["m_eff"])
    half, full = torch.polar(torch.ones_like(theta), -theta / 2), torch.polar(torch.ones_like(theta), -theta)
    cell = spacing ** 2

    def reservoir(f, rho):
        r1 = _res_rates(f, rho, pump, p)
        r2 = _res_rates([n + 0.25 * dt * r for n, r in zip(f, r1)], rho, pump, p)
        return [(n + 0.5 * dt * r).clamp_min(0) for n, r in zip(f, r2)]

    def local(y, f):
        v = pot + 0j if not torch.is_tensor(pot) else pot
        vre, vim = (v.real, v.imag) if torch.is_tensor(v) and v.is_complex() else (v.real if torch.is_tensor(v) else 0.0, 0.0)
        gain = 0.5 * (p["R"] * f[0] - p["gamma_C"]) + vim / p["hbar"]
        x = 2 * gain * dt
        time = dt * torch.where(x.abs() < 1e-6, 1 + x / 2 + x * x / 6, torch.expm1(x) / torch.where(x == 0, torch.ones_like(x), x))
        phase = ((vre + _potential_energy(f, p)) * dt + p["g_C"] * _density(y) * time) / p["hbar"]
        return y * torch.polar(torch.exp(gain * dt), -phase)

    if kouter:
        spec = torch.fft.fft2(psi) * half
        for k in range(steps):
            y = torch.fft.ifft2(spec)
            fields = reservoir(fields, _density(y))
            y = local(y, fields)
            fields = reservoir(fields, _density(y))
            if seeds is not None:
                y = _wigner(y, fields[0], k, seeds, p, dt, cell, double)
            spec = torch.fft.fft2(y) * full
        return spec * half.conj(), fields
    for k in range(steps):
        fields = reservoir(fields, _density(psi))
        psi = local(torch.fft.ifft2(torch.fft.fft2(psi) * half), fields)
        if seeds is not None:
            psi = _wigner(psi, fields[0], k, seeds, p, dt, cell, double)
        psi = torch.fft.ifft2(torch.fft.fft2(psi) * half)
        fields = reservoir(fields, _density(psi))
    return psi, fields


RK4 = ([[], [0.5], [0, 0.5], [0, 0, 1.0]], [1 / 6, 1 / 3, 1 / 3, 1 / 6], [0, 0.5, 0.5, 1.0])
DP5 = ([[], [1 / 5], [3 / 40, 9 / 40], [44 / 45, -56 / 15, 32 / 9],
        [19372 / 6561, -25360 / 2187, 64448 / 6561, -212 / 729],
        [9017 / 3168, -355 / 33, 46732 / 5247, 49 / 176, -5103 / 18656],
        [35 / 384, 0, 500 / 1113, 125 / 192, -2187 / 6784, 11 / 84]],
       [35 / 384, 0, 500 / 1113, 125 / 192, -2187 / 6784, 11 / 84, 0], [0, 1 / 5, 3 / 10, 4 / 5, 8 / 9, 1.0, 1.0])


def _lawson_exact(psi, fields, pump, pot, p, spacing, h, steps, seeds, tableau, spinor):
    weights, b, c = tableau
    kx, ky = _k_axes(psi.shape[-1], psi.shape[-2], spacing)
    k2 = kx ** 2 + ky ** 2
    energy = p["hbar"] ** 2 / (2 * p["m_eff"]) * k2
    if spinor:
        z = 0.5 * p["zeeman"]
        u = torch.complex(p["te_tm"] * (kx ** 2 - ky ** 2), -2 * p["te_tm"] * kx * ky)
        omega = torch.sqrt(z * z + _density(u))

    def linear(spec, tau):
        if tau == 0:
            return spec
        common = torch.polar(torch.ones_like(energy), -energy * tau / p["hbar"])
        if not spinor:
            return spec * common
        angle = omega * tau / p["hbar"]
        s = torch.where(omega > 0, torch.sin(angle) / torch.where(omega > 0, omega, torch.ones_like(omega)),
                        torch.full_like(omega, tau / p["hbar"]))
        cos, up, down = torch.cos(angle), spec[:, 0], spec[:, 1]
        return common * torch.stack([(cos - 1j * s * z) * up - 1j * s * u * down,
                                     -1j * s * u.conj() * up + (cos + 1j * s * z) * down], 1)

    share = 0.5 if spinor else 1.0
    for k in range(steps):
        spec0 = torch.fft.fft2(psi)
        rhs_k, rates = [], []
        for i, row in enumerate(weights):
            spec, f = linear(spec0, c[i] * h), list(fields)
            for j, a in enumerate(row):
                if a:
                    spec = spec + h * a * linear(rhs_k[j], (c[i] - c[j]) * h)
                    f = [n + h * a * r for n, r in zip(f, rates[j])]
            y = torch.fft.ifft2(spec)
            rho = _density(y)
            energy_r = p["g_C"] * rho + _potential_energy(f, p) + pot
            if spinor:
                energy_r = energy_r + p["alpha_2"] * rho.flip(1)
            gain = 0.5 * (p["R"] * f[0] - p["gamma_C"])
            rhs_k.append(torch.fft.fft2((gain - 1j / p["hbar"] * energy_r) * y))
            rates.append(_res_rates(f, rho, share * pump, p))
        spec = linear(spec0, h)
        for j, w in enumerate(b):
            if w:
                spec = spec + h * w * linear(rhs_k[j], (1 - c[j]) * h)
                fields = [n + h * w * r for n, r in zip(fields, rates[j])]
        fields = [n.clamp_min(0) for n in fields]
        psi = torch.fft.ifft2(spec)
        if seeds is not None:
            psi = _wigner(psi, fields[0], k, seeds, p, h, spacing ** 2, False)
    return psi, fields


def _grid_exact(case, seed):
    x = _inputs(case, seed)
    p, kind = _physics(case), case["kind"]
    env = x["env"]
    if kind == "dropin":
        _, _, r2 = _radius2(case["nx"], case["ny"], case["spacing"])
        env = torch.exp(-0.5 * r2 / (0.12 * case["spacing"] * min(case["nx"], case["ny"])) ** 2).to(_real(case))
    pump = env.double() * P0
    psi = x["psi"].to(torch.complex128)
    two = case.get("reservoir") == "double" or kind == "dp5"
    fields = [f.double() for f in x["res"]] if two else [x["res"].double()]
    pot = 0.0 if x["pot"] is None else x["pot"].to(torch.complex128) if x["pot"].is_complex() else x["pot"].double()
    seeds = x["seeds"] if case.get("noise") else None
    double = case.get("precision") == "double"
    rest = (p, case["spacing"], case.get("dt", case.get("h")), case["steps"], seeds)
    if kind in ("rk4", "dropin"):
        psi, fields = _rk4_exact(psi, fields, pump, pot, *rest, double)
    elif kind in ("split0", "split1"):
        psi, fields = _split_exact(psi, fields, pump, pot, *rest, double, kind == "split1")
    else:
        psi, fields = _lawson_exact(psi, fields, pump, pot, *rest, RK4 if kind == "ifrk4" else DP5, kind == "dp5")
    return {"psi": psi, "res": torch.stack(fields) if two else fields[0]}


def _sweep_exact(case, seed):
    x = _sweep_inputs(case, seed)
    psi, res, at = [], [], 0
    for m, n in enumerate(x["sizes"]):
        shape = (1, 1, n, n)
        y, f = _rk4_exact(x["psi"][at:at + n * n].reshape(shape).to(torch.complex128),
                          [x["res"][at:at + n * n].reshape(shape).double()], x["envs"][m].double() * P0, 0.0,
                          PHYSICS, 0.5, case["dt"], case["steps"], [x["seeds"][m]] if case["noise"] else None, False)
        psi.append(y.reshape(-1))
        res.append(f[0].reshape(-1))
        at += n * n
    return {"psi": torch.cat(psi), "res": torch.cat(res)}


def _fno_exact(case, seed):
    n, m, w = case["n"], case["modes"], case["width"]
    a, target = (t.double() for t in _fno_inputs(case, seed))
    p = {k: torch.tensor(v.astype(np.float32).astype(np.float64), device=_device(), requires_grad=True)
         for k, v in _fno_params(case, seed).items()}
    grid = torch.arange(n, dtype=torch.float64, device=_device())
    rows = torch.cat([torch.arange(m), torch.arange(n - m, n)]).double().to(_device())
    kept = torch.arange(m, dtype=torch.float64, device=_device())
    fx = torch.exp(-2j * math.pi * torch.outer(grid, kept) / n)
    gy = torch.exp(-2j * math.pi * torch.outer(rows, grid) / n)
    fold = torch.where(kept == 0, 1.0, 2.0).double() / (n * n)

    def gelu(v):
        return torch.nn.functional.gelu(v, approximate="tanh")

    def mix(weight, bias, v):
        return torch.einsum("oi,bihw->bohw", weight, v) + bias[:, None, None]

    v = mix(p["lift_w"], p["lift_b"], a)
    for k in range(case["layers"]):
        spec = torch.einsum("ry,biyk->birk", gy, v.to(torch.complex128) @ fx)
        spec = torch.einsum("birk,rkio->bork", spec, torch.complex(p[f"spec{k}_re"], p[f"spec{k}_im"]))
        back = torch.einsum("ry,bork->boyk", gy.conj(), spec * fold) @ fx.conj().T
        v = back.real + mix(p[f"w{k}"], p[f"b{k}"], v)
        v = gelu(v) if k < case["layers"] - 1 else v
    out = mix(p["proj2_w"], p["proj2_b"], gelu(mix(p["proj1_w"], p["proj1_b"], v)))
    loss = ((out - target) ** 2).mean()
    loss.backward()
    return {"out": out.detach(), "loss": float(loss.detach()), "grads": {k: t.grad for k, t in p.items()}}


def exact(case, seed):
    if case["kind"] == "fno":
        return _fno_exact(case, seed)
    if case["kind"] == "sweep":
        return _sweep_exact(case, seed)
    return _grid_exact(case, seed)
