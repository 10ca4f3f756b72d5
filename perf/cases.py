"""The performance cases of this framework: what its users have it do, through the entry points they call.

Four kinds of work, each over the sizes its users bring:

* the DP Langevin integrator (`Batch` of `dp_model`, `percolation_dornic_2d`, `critical_exp_theta_delta`):
  single runs and small ensembles in FP64, the reference's precision; ragged parameter sweeps in FP32;
* the three-field Rietkerk integrator (`Batch` of `rietkerk_model`), noise on and off, FP32 and FP64;
* what a study does beside the integration: the consumer's movement (`fke_advdiff`) and the pattern's
  power spectrum (`Batch.power_spectrum`);
* the surrogate network (`surrogate.MLP`) that guides the search for the critical point.

A pass of an integrator case starts from the same uploaded state, advances it with its measurements and
hands back the whole final state, the observables and the status words.
"""
import math

import numpy as np
import torch

import trophic_maelstorm_gb300 as tmg
from trophic_maelstorm_gb300 import _lib, api
from trophic_maelstorm_gb300 import surrogate as sg

_CTX = None


def _ctx():
    """The one context a program keeps."""
    global _CTX
    if _CTX is None:
        _CTX = tmg.Context(0)
    return _CTX


# ------------------------------------------------------------------------------------------ the cases
def listed():
    return [
        # one run of the reference's own call: 128 x 128, FP64, a ramped 0.72 -> 0.70, t = 20
        {"name": "dp_call_f64_128", "kind": "call", "L": 128, "reps": 1, "t_max": 20.0, "a": 0.72, "a_end": 0.70},
        # spreading from one seed at the centre, FP64: many steps of almost empty lattices, latency alone
        {"name": "dp_spread_f64_101", "kind": "spread", "L": 101, "div": 4, "reps": 16, "t_max": 20.0},
        # an FP64 ensemble as the multi-species code integrates it: RK4 remainder, Gaussian above 100, clamp
        {"name": "dp_f64_256x16_rk4", "kind": "dp", "L": 256, "ragged": False, "reps": 16, "n_a": 1, "precision": "f64",
         "steps": 32, "meas": 2, "occupied": 1.0, "remainder": "rk4", "sampler": "gauss100"},
        # the finite-size sweep: five sides x replicates x 16 values of a in one ragged FP32 batch, fully active
        {"name": "dp_f32_sweep", "kind": "dp", "L": 1024, "ragged": True, "reps": 4, "n_a": 16, "precision": "f32",
         "steps": 40, "meas": 2, "occupied": 1.0, "remainder": "euler", "sampler": "exact"},
        # the late, dilute stretch of a near-critical run (most of a long sweep's steps), measured on the way
        {"name": "dp_f32_dilute_512x32", "kind": "dp", "L": 512, "ragged": False, "reps": 8, "n_a": 4,
         "precision": "f32", "steps": 100, "meas": 4, "occupied": 0.2, "remainder": "euler", "sampler": "exact"},
        # one large Rietkerk lattice, FP32, from the uniform random start
        {"name": "rk_f32_4096", "kind": "rietkerk", "L": 4096, "reps": 1, "precision": "f32", "steps": 24,
         "meas": 1, "start": "random", "noise": True, "R": 0.9},
        # a small ensemble of vegetated lattices (the pattern study), FP32: too small to fill the GPU for long
        {"name": "rk_f32_256x8", "kind": "rietkerk", "L": 256, "reps": 8, "precision": "f32", "steps": 100,
         "meas": 2, "start": "vegetated", "noise": True, "R": 1.2},
        # part of the rainfall sweep in the reference's precision
        {"name": "rk_f64_256x16", "kind": "rietkerk", "L": 256, "reps": 16, "precision": "f64", "steps": 20,
         "meas": 1, "start": "random", "noise": True, "R": 1.0},
        # the noise-off Rietkerk step on an odd side, FP64 (the mean-field reference runs)
        {"name": "rk_off_f64_301x2", "kind": "rietkerk", "L": 301, "reps": 2, "precision": "f64", "steps": 20,
         "meas": 0, "start": "vegetated", "noise": False, "R": 1.2},
        # one movement of a consumer field, FP64, on the workspace that a step loop keeps
        {"name": "fke_f64_1024", "kind": "fke", "L": 1024, "precision": "f64", "D": 1.0, "v": 1.0, "vmax": 1.0},
        # the surrogate's fit on a corpus of 200 runs x 60 times, and the proposal's grid of predictions
        {"name": "mlp_fit_12000", "kind": "mlp", "n": 12000, "steps": 50, "n_predict": 1201},
        # the wavelength estimate of one pattern frame
        {"name": "spectrum_f64_512", "kind": "spectrum", "L": 512, "precision": "f64", "binwidth": 0.5},
    ]


def _log(rng, lo, hi):
    """A whole number spread over the logarithm of [lo, hi]."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 0.5)))))))


def draw(rng):
    kind = rng.choice(["call", "spread", "dp", "dp", "dp", "rietkerk", "rietkerk", "off", "fke", "mlp", "spectrum"])
    if kind == "call":
        L = _log(rng, 24, 160)
        a = round(rng.uniform(0.5, 0.74), 4)
        return {"kind": "call", "L": L, "reps": _log(rng, 1, max(1, 32768 // (L * L))), "t_max": rng.choice([5.0, 10.0, 20.0]),
                "a": a, "a_end": round(a - rng.choice([0.0, 0.02]), 4)}
    if kind == "spread":
        return {"kind": "spread", "L": _log(rng, 33, 160), "div": rng.randint(1, 4), "reps": _log(rng, 1, 16),
                "t_max": rng.choice([5.0, 10.0, 20.0])}
    if kind == "dp":
        precision = rng.choice(["f64", "f32", "f32"])
        top = 1 << 20 if precision == "f64" else 1 << 25      # sites of the largest drawn batch
        ragged = rng.random() < 0.3
        L = _log(rng, 48, 1024 if precision == "f32" else 512)
        n_a = rng.choice([1, 2, 4, 8])
        sites = L * L * n_a * (1.4 if ragged else 1.0)
        return {"kind": "dp", "L": L, "ragged": ragged, "reps": _log(rng, 1, max(1, min(32, int(top / sites)))), "n_a": n_a,
                "precision": precision, "steps": rng.choice([16, 33, 64] if precision == "f32" else [8, 33]), "meas": rng.randint(1, 4),
                "occupied": rng.choice([1.0, 1.0, 0.5, 0.1]), "remainder": rng.choice(["euler", "euler", "rk4"]),
                "sampler": rng.choice(["exact", "exact", "gauss100"])}
    if kind in ("rietkerk", "off"):
        precision = rng.choice(["f64", "f32", "f32"])
        L = _log(rng, 48, 2048 if precision == "f32" else 400)
        top = 1 << 22 if precision == "f32" else 1 << 19
        return {"kind": "rietkerk", "L": L, "reps": _log(rng, 1, max(1, min(16, top // (L * L)))), "precision": precision,
                "steps": rng.choice([10, 33, 64] if precision == "f32" else [5, 20]), "meas": rng.randint(0, 2),
                "start": rng.choice(["random", "vegetated"]), "noise": kind == "rietkerk",
                "R": round(rng.uniform(0.6, 1.3), 3)}
    if kind == "fke":
        return {"kind": "fke", "L": _log(rng, 32, 1024), "precision": rng.choice(["f64", "f64", "f32"]),
                "D": rng.choice([0.3, 1.0, 2.0]), "v": rng.choice([0.5, 1.0, 3.0]), "vmax": rng.choice([0.5, 1.0, 4.0])}
    if kind == "mlp":
        return {"kind": "mlp", "n": _log(rng, 100, 20000), "steps": rng.randint(5, 50), "n_predict": _log(rng, 1, 20000)}
    return {"kind": "spectrum", "L": _log(rng, 32, 700), "precision": rng.choice(["f64", "f32"]),
            "binwidth": rng.choice([0.5, 1.0])}


# ------------------------------------------------------------------------------------------ their inputs
def _prec(case):
    return (tmg.TM_FP64, torch.float64) if case["precision"] == "f64" else (tmg.TM_FP32, torch.float32)


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _uniform(gen, shape, lo, hi, dtype=torch.float64):
    return torch.rand(shape, generator=gen, device="cuda", dtype=dtype) * (hi - lo) + lo


def _sides(case):
    if not case["ragged"]:
        return [case["L"]]
    return [max(8, case["L"] >> k) for k in range(4, -1, -1)]


def _dp_instances(case, seed):
    """(L, a, replicate) in that order: a log-spaced within 2 % of the critical point, one Philox key each."""
    Ls, av = [], []
    for L in _sides(case):
        for i in range(case["n_a"]):
            a = 0.53 * 0.98 * (1.02 / 0.98) ** (i / max(1, case["n_a"] - 1)) if case["n_a"] > 1 else 0.53
            Ls += [L] * case["reps"]
            av += [a] * case["reps"]
    return tmg.instances(Ls, [seed * 1000003 + k for k in range(len(Ls))], np.array(av))


def _dp_field(gen, L, occupied, dtype):
    """Fully active: 1 + U(-0.01, 0.01).  Else occupied patches of 8 x 8 sites, 0.05 to 0.6 where a site is occupied."""
    if occupied >= 1.0:
        return _uniform(gen, (L, L), 0.99, 1.01, dtype)
    n = (L + 7) // 8
    patch = (torch.rand((n, n), generator=gen, device="cuda") < occupied).repeat_interleave(8, 0).repeat_interleave(8, 1)
    keep = patch[:L, :L] & (torch.rand((L, L), generator=gen, device="cuda") < 0.6)
    return _uniform(gen, (L, L), 0.05, 0.6, dtype) * keep


def _rk_field(gen, L, start, R, dtype):
    """[P, W, O]: P ~ U(0, 1), W = 0.5, O = 1, or the vegetated fixed point with P perturbed by 10 %."""
    if start == "random":
        return torch.stack([_uniform(gen, (L, L), 0.0, 1.0, dtype), torch.full((L, L), 0.5, device="cuda", dtype=dtype),
                            torch.full((L, L), 1.0, device="cuda", dtype=dtype)])
    m = tmg.rietkerk_model()
    W = m.d * m.k1 / (m.c * m.gmax - m.d)
    P = max(0.5, (R - m.rW * W) * m.c / m.d)
    O = R / (m.alpha * (P + m.k2 * m.W0) / (P + m.k2))
    one = torch.ones((L, L), device="cuda", dtype=dtype)
    return torch.stack([P * _uniform(gen, (L, L), 0.9, 1.1, dtype), W * one, O * one])


def _meas(case):
    """Measurement steps of a pass: evenly spread, the last at its end."""
    n, m = case["steps"], case["meas"]
    return [max(1, n * (j + 1) // m) for j in range(m)]


def _batch_state(case, seed):
    gen = _gen(seed)
    prec, dtype = _prec(case)
    if case["kind"] == "dp":
        inst = _dp_instances(case, seed)
        model = tmg.dp_model(b=2.0, D=1.0, sigma=1.0, dt=0.1, clamp_eps=1e-12 if case["remainder"] == "rk4" else 0.0,
                             clamp_lo=-1e-80 if case["remainder"] == "rk4" else 0.0,
                             remainder=_lib.TM_REM_RK4 if case["remainder"] == "rk4" else _lib.TM_REM_EULER_EXACT,
                             sampler=_lib.TM_SAMPLER_REF_GAUSS100 if case["sampler"] == "gauss100" else _lib.TM_SAMPLER_EXACT)
        frames = [_dp_field(gen, i.L, case["occupied"], dtype) for i in inst]
    else:
        inst = tmg.instances([case["L"]] * case["reps"], [seed * 1000003 + k for k in range(case["reps"])],
                             case["R"] * (1.0 + 0.01 * np.arange(case["reps"])))
        model = tmg.rietkerk_model(deterministic=0 if case["noise"] else 1)
        frames = [_rk_field(gen, case["L"], case["start"], i.a, dtype) for i in inst]
    batch = tmg.Batch(_ctx(), model, inst, prec)
    total, off, fs = api.layout(inst, batch.nf)
    init = torch.zeros(total, device="cuda", dtype=dtype)
    for k, f in enumerate(frames):
        n = inst[k].L * inst[k].L
        for j, part in enumerate(f.reshape(batch.nf, n)):
            init[int(off[k] + j * fs[k]):int(off[k] + j * fs[k]) + n] = part
    return {"batch": batch, "init": init, "out": torch.empty_like(init), "meas": _meas(case)}


def _call_seed(seed):
    return (seed * 2654435761) & 0x7FFFFFFF


def _mlp_data(case, seed):
    """Normalised (a, log L, log t) and targets as the fit of a corpus has them: a decay in t that bends with a."""
    rng = np.random.default_rng(seed)
    n = case["n"]
    x = np.stack([rng.uniform(-1, 1, n), rng.integers(-2, 3, n) / 2.0, rng.uniform(-1, 1, n)], 1).astype(np.float32)
    y0 = -0.45 * 1.5 * (x[:, 2] + 1) + 0.6 * x[:, 0] * (x[:, 2] + 1) + 0.02 * rng.standard_normal(n)
    y1 = 1.0 / (1.0 + np.exp(3.0 * (x[:, 2] - 0.5) - 2.0 * x[:, 0] - x[:, 1]))
    w = np.stack([(rng.random(n) < 0.95).astype(np.float32), np.ones(n, np.float32)], 1)
    grid = np.stack([np.linspace(-1, 1, case["n_predict"]), np.zeros(case["n_predict"]), np.ones(case["n_predict"])],
                    1).astype(np.float32)
    return x, np.stack([y0, y1], 1).astype(np.float32), w, grid


def _fke_fields(case, seed):
    gen = _gen(seed)
    _, dtype = _prec(case)
    L = case["L"]
    rho = _uniform(gen, (L, L), 0.0, 2.0, dtype) * (torch.rand((L, L), generator=gen, device="cuda") > 0.3)
    return (rho, _uniform(gen, (L, L), 0.0, 1.0, dtype), _uniform(gen, (L, L), -case["vmax"], case["vmax"], dtype),
            _uniform(gen, (L, L), -case["vmax"], case["vmax"], dtype))


def _spectrum_frame(case, seed):
    """A pattern of about ten wavelengths with noise."""
    gen = _gen(seed)
    L = case["L"]
    x = torch.arange(L, device="cuda", dtype=torch.float64) * (2 * math.pi / L)
    ph = _uniform(gen, (3,), 0.0, 6.0)
    f = sum(torch.cos(kx * x[None, :] + ky * x[:, None] + ph[i]) for i, (kx, ky) in enumerate([(11, 0), (5, 9), (-6, 9)]))
    return (f + 3.0 + _uniform(gen, (L, L), 0.0, 1.0)).to(_prec(case)[1])


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case, "kind": kind}
    if kind in ("dp", "rietkerk"):
        s.update(_batch_state(case, seed))
    elif kind == "call":
        rng = np.random.default_rng(seed)
        s.update(frame=1.0 + rng.uniform(-0.01, 0.01, case["L"] ** 2), seed=_call_seed(seed), ctx=_ctx(),
                 t_meas=tmg.logarithm10_time_bins(case["t_max"], 0.1))
    elif kind == "spread":
        s.update(seed=_call_seed(seed), ctx=_ctx())
    elif kind == "fke":
        prec, _ = _prec(case)
        s.update(fields=_fke_fields(case, seed), prec=prec, params=tmg.fke_parameters(case["D"], case["v"], 1.0, 1.5),
                 workspace=api.fke_workspace(case["L"], prec))
    elif kind == "mlp":
        x, y, w, grid = _mlp_data(case, seed)
        params = sg.init_params(seed)
        net = sg.MLP(_ctx(), params)
        net.set_data(x, y, w)
        s.update(net=net, params=params, grid=grid)
    else:
        prec, dtype = _prec(case)
        inst = tmg.instances([case["L"]], [1], 0.53)
        batch = tmg.Batch(_ctx(), tmg.dp_model(), inst, prec)
        total, _, _ = api.layout(inst, 1)
        buf = torch.zeros(total, device="cuda", dtype=dtype)
        buf[:case["L"] ** 2] = _spectrum_frame(case, seed).reshape(-1)
        torch.cuda.synchronize()
        batch.upload_device(buf.data_ptr())
        s.update(batch=batch)
    torch.cuda.synchronize()
    return s


# ------------------------------------------------------------------------------------------ one pass
def run(s):
    case, kind = s["case"], s["kind"]
    if kind in ("dp", "rietkerk"):
        b = s["batch"]
        b.upload_device(s["init"].data_ptr())
        obs, status = b.advance(case["steps"], s["meas"])
        _lib.check(_lib.lib().tm_batch_download_device(b.handle, s["out"].data_ptr()), "tm_batch_download_device")
        return {"state": s["out"], "obs": obs, "status": status.astype(np.int64)}
    if kind == "call":
        rows, status = tmg.percolation_dornic_2d(s["t_meas"], s["frame"], case["t_max"], case["a"], 2.0, 1.0, 1.0, 0.1, 1.0,
                                                 case["reps"], case["L"], seed=s["seed"], a_end=case["a_end"], ctx=s["ctx"])
        return {"rows": rows, "status": status.astype(np.int64)}
    if kind == "spread":
        rows, status = tmg.critical_exp_theta_delta(None, case["div"], case["t_max"], 0.53, 2.0, 1.0, 1.0, 0.1, 1.0,
                                                    case["reps"], case["L"], seed=s["seed"], ctx=s["ctx"])
        return {"rows": rows, "status": status.astype(np.int64)}
    if kind == "fke":
        return tmg.fke_advdiff(*s["fields"], s["params"], precision=s["prec"], workspace=s["workspace"])
    if kind == "mlp":
        net = s["net"]
        net.set_params(s["params"])
        y = net.predict(s["grid"])
        loss, grad = net.loss_grad()
        hist = net.train(case["steps"], lr=1e-3)
        return {"y": y, "loss": loss, "grad": grad, "hist": hist, "params": net.get_params(), "y_fit": net.predict(s["grid"])}
    k, power = s["batch"].power_spectrum(0, 0, case["binwidth"])
    return {"k": k, "power": power}


# ------------------------------------------------------------------------------------------ what it needs
L2_BYTES = 129e6                     # a state that fits here may stay on the chip between the steps of a pass


def _step_bytes(sites, nf, e, steps):
    """A state's values read and written: once a pass where it fits the last-level cache, else once a step."""
    once = 2.0 * sites * nf * e
    return once if once <= L2_BYTES else once * steps


def work(case):
    kind = case["kind"]
    if kind == "dp":
        sites = float(sum(i.L * i.L for i in _dp_instances(case, 0)))
        e = 8 if case["precision"] == "f64" else 4
        # neighbour sum and constants 8, Poisson-Gamma draw 40, remainder 4 (12 with RK4)
        return {"bytes": _step_bytes(sites, 1, e, case["steps"]),
                "flops": sites * case["steps"] * (60 if case["remainder"] == "rk4" else 52)}
    if kind == "rietkerk":
        sites = float(case["reps"] * case["L"] ** 2)
        e = 8 if case["precision"] == "f64" else 4
        # four stages of two (three) Laplacians and the reactions 36, their sums 10; the draw of P 48
        return {"bytes": _step_bytes(sites, 3, e, case["steps"]),
                "flops": sites * case["steps"] * (4 * 46 + (48 if case["noise"] else 24))}
    if kind in ("call", "spread"):
        n = case["reps"] * (case["div"] if kind == "spread" else 1)
        sites = float(n * case["L"] ** 2)
        live = math.pi * 400.0 / case["L"] ** 2 if kind == "spread" else 1.0        # a seed's cluster at t = 20
        return {"bytes": _step_bytes(sites, 1, 8, 1), "flops": sites * min(1.0, live) * 10 * case["t_max"] * 52}
    if kind == "fke":
        n = float(case["L"] ** 2)
        p = tmg.fke_parameters(case["D"], case["v"], 1.0, 1.5)
        taps = 2 * p.RD + 1 + 2 * p.RV + 1
        return {"bytes": 5 * n * (8 if case["precision"] == "f64" else 4), "flops": n * (2 * 3 * taps + 10)}
    if kind == "mlp":
        fwd = 2.0 * (3 * 128 + 2 * 128 * 128 + 128 * 2)
        passes = case["steps"] + 1
        return {"bytes": passes * (case["n"] * 28.0 + 4 * 33794 * 4) + case["n_predict"] * 40.0,
                "flops": fwd * (3 * passes * case["n"] + 2 * case["n_predict"])}
    n = float(case["L"] ** 2)
    return {"bytes": n * (8 if case["precision"] == "f64" else 4), "flops": 2.5 * n * math.log2(n) + 4 * n}


# ------------------------------------------------------------------------------------------ 64-bit results
def _exact_rietkerk_off(case, seed):
    """The noise-off three-field RK4 step on whole lattices."""
    gen = _gen(seed)
    m = tmg.rietkerk_model()
    nf, L = 3, case["L"]
    fs = (L * L + 31) // 32 * 32
    dtype = _prec(case)[1]
    R = case["R"] * (1.0 + 0.01 * np.arange(case["reps"]))
    out = torch.zeros(case["reps"] * nf * fs, device="cuda", dtype=torch.float64)
    obs = np.zeros((case["meas"], case["reps"], 4))

    def lap(a):
        return a.roll(1, 0) + a.roll(-1, 0) + a.roll(1, 1) + a.roll(-1, 1) - 4.0 * a

    def rhs(u, r):
        P, W, O = u
        infil = m.alpha * (P + m.k2 * m.W0) / (P + m.k2) * O
        upt = m.gmax * W * P / (W + m.k1)
        return torch.stack([m.c * upt - m.d * P + m.DP * lap(P), infil - upt - m.rW * W + m.DW * lap(W),
                            r - infil + m.DO * lap(O)])

    at = _meas(case)
    for k in range(case["reps"]):
        u = _rk_field(gen, L, case["start"], R[k], dtype).double()
        for step in range(1, case["steps"] + 1):
            k1 = rhs(u, R[k])
            k2 = rhs(u + m.dt / 2 * k1, R[k])
            k3 = rhs(u + m.dt / 2 * k2, R[k])
            k4 = rhs(u + m.dt * k3, R[k])
            u = u + m.dt / 6 * (k1 + 2 * k2 + 2 * k3 + k4)
            u = torch.where((u < m.clamp_eps) & (u >= m.clamp_lo), torch.zeros_like(u), u)
            for j, t in enumerate(at):
                if t == step:
                    obs[j, k] = [float(u[0].mean()), float(u[1].mean()), float(u[2].mean()), float((u[0] > 0).sum())]
        for f in range(nf):
            out[(k * nf + f) * fs:(k * nf + f) * fs + L * L] = u[f].reshape(-1)
    return {"state": out, "obs": obs, "status": np.zeros(case["reps"], np.int64)}


def _exact_fke(case, seed):
    """Every source's mass scattered through the four stencils, in 64 bits."""
    rho, g, vx, vy = (t.double() for t in _fke_fields(case, seed))
    p = tmg.fke_parameters(case["D"], case["v"], 1.0, 1.5)
    L = case["L"]
    if case["precision"] == "f32":                       # the shift is a rounding of this precision's product
        pref = torch.tensor(p.pref, dtype=torch.float32, device="cuda")
        i = torch.arange(L, device="cuda", dtype=torch.float32)
        mx, my = i[:, None] + vx.float() * pref, i[None, :] + vy.float() * pref
    else:
        i = torch.arange(L, device="cuda", dtype=torch.float64)
        mx, my = i[:, None] + vx * p.pref, i[None, :] + vy * p.pref
    far = torch.trunc(mx + torch.copysign(torch.full_like(mx, 0.5), mx)), torch.trunc(my + torch.copysign(torch.full_like(my, 0.5), my))
    mx, my = (t.long() for t in far)
    rho = torch.where(rho < 1e-10, torch.zeros_like(rho), rho)
    n = torch.arange(L, device="cuda")
    ci, cj = n[:, None].expand(L, L), n[None, :].expand(L, L)
    out = torch.zeros(L * L, device="cuda", dtype=torch.float64)
    for w, ri, gi, rj, gj in ((g * g * rho, ci, p.gD, cj, p.gD), (g * (1 - g) * rho, ci, p.gD, my, p.gV),
                              (g * (1 - g) * rho, mx, p.gV, cj, p.gD), ((1 - g) ** 2 * rho, mx, p.gV, my, p.gV)):
        for a in range(-(len(gi) - 1), len(gi)):
            row = (ri + a) % L * L
            for b in range(-(len(gj) - 1), len(gj)):
                out.index_add_(0, (row + (rj + b) % L).reshape(-1), (w * (gi[abs(a)] * gj[abs(b)])).reshape(-1))
    return out.reshape(L, L)


def _exact_mlp(case, seed):
    """The network on its BF16 weights with activations and gradients in 64 bits."""
    x, y, w, grid = (torch.from_numpy(t).double() for t in _mlp_data(case, seed))
    p = torch.from_numpy(sg.init_params(seed))
    parts, at = [], 0
    for shape in ((128, 3), (128,), (128, 128), (128,), (128, 128), (128,), (2, 128), (2,)):
        n = int(np.prod(shape))
        q = p[at:at + n].reshape(shape)
        parts.append((q.bfloat16() if len(shape) == 2 else q).double().requires_grad_())
        at += n

    def net(f):
        for k in (0, 2, 4):
            f = torch.nn.functional.gelu(f @ parts[k].T + parts[k + 1], approximate="tanh")
        return f @ parts[6].T + parts[7]

    loss = (w * (net(x) - y) ** 2).sum() / case["n"]
    grads = torch.autograd.grad(loss, parts)
    with torch.no_grad():
        out = net(grid)
    return {"y": out, "loss": float(loss.detach()), "grad": torch.cat([t.reshape(-1) for t in grads])}


def _exact_spectrum(case, seed):
    """|FFT|^2 of the frame over its maximum, averaged over annuli, times their area."""
    f = _spectrum_frame(case, seed).double().cpu().numpy()
    L, bw = case["L"], case["binwidth"]
    p = np.abs(np.fft.fft2(f / f.max())) ** 2
    fr = np.fft.fftfreq(L) * L
    k = np.sqrt(fr[:, None] ** 2 + fr[None, :] ** 2).reshape(-1)
    e = np.arange(1 - bw / 2, L // 2 + 1, bw)
    total, _ = np.histogram(k, e, weights=p.reshape(-1))
    count, _ = np.histogram(k, e)
    power = np.where(count > 0, total / np.maximum(count, 1), 0.0) * math.pi * (e[1:] ** 2 - e[:-1] ** 2)
    return {"k": 0.5 * (e[1:] + e[:-1]), "power": power}


def exact(case, seed):
    kind = case["kind"]
    if kind == "rietkerk" and not case["noise"]:
        return _exact_rietkerk_off(case, seed)
    if kind == "fke":
        return _exact_fke(case, seed)
    if kind == "mlp":
        return _exact_mlp(case, seed)
    if kind == "spectrum":
        return _exact_spectrum(case, seed)
    return None                      # a noisy run has no value but the one its own random stream gives
