"""Performance cases: the calls a user of this package makes, over the range of sizes they are made at.

Kinds (each through the public entry points, lib.Context, lib.Network, forward.ClaritasForwardModel):

  trace     photons through a built scene: the full scene, the small disc-beam scene, the dense weighted one,
            and the reference's own random stream with per-ray records
  build     a scene's tables (set_scene, build_particles) and their read-back
  sweep     many scenarios built and traced together, as the surrogate's training data and the concentration
            inversion are made
  simulate  the reference's whole call: a model object, a named material, a photon count
  predict   the surrogate network on a batch of queries
  train     one epoch of the surrogate's training

Monte Carlo tallies have no closed value: exact() is None for them.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from tardiis_and_claritas_gb300 import abi, forward as F, lib as L, scene as S, surrogate as G

# FP32-equivalent operations per launched photon of each traced scene (the package's published work table times
# the event counts of a trace)
OPS_PER_PHOTON = {"full": 1665.0, "disc": 2425.0, "dense": 58300.0, "parity": 1712.0, "sweep": 1772.0,
                  "simulate": 3000.0}
MLP_FLOP = 2 * (6 * 256 + 3 * 256 * 256 + 256 * 3)  # per query
MLP_PARAMS = L.Network.N_PARAMS


def listed():
    return [
        # one quick answer from the small scene: what an interactive call or a test asks for
        {"name": "trace_disc_1e5", "kind": "trace", "scene": "disc", "photons": 100_000},
        # the benchmark's step: the full scene at 1e8 photons
        {"name": "trace_full_1e8", "kind": "trace", "scene": "full", "photons": 100_000_000},
        # the full scene at a photon count of an ordinary run
        {"name": "trace_full_2e6", "kind": "trace", "scene": "full", "photons": 2_000_000},
        # optically dense clay with weights and Russian roulette: few photons, long histories
        {"name": "trace_dense_5e4", "kind": "trace", "scene": "dense", "photons": 50_000},
        # the reference's random stream with per-ray records: the parity and per-ray output path
        {"name": "trace_records_131072", "kind": "trace", "scene": "parity", "photons": 131_072},
        # tables of one scene with a supplied (r, z) field, in the reference's order of operations: every new
        # concentration or particle population rebuilds them
        {"name": "build_grid_63", "kind": "build", "field": "grid", "bins": 63, "angles": 1801, "fast": False,
         "max_um": 274.0},
        # the reference's default sediment model: the meridional field solved for every size bin
        {"name": "build_meridional_64", "kind": "build", "field": "meridional", "bins": 64, "angles": 1801,
         "fast": False, "max_um": 200.0},
        # Monte Carlo labels for the surrogate: scenarios of 1e6 photons, tables built fast
        {"name": "sweep_128x1e6", "kind": "sweep", "scenarios": 128, "photons": 1_000_000},
        # the reference's whole call with a named material, batches and path provenance included
        {"name": "simulate_loess_5e5", "kind": "simulate", "material": "loess", "photons": 500_000},
        # one scenario's concentration search (401 candidates)
        {"name": "predict_401", "kind": "predict", "queries": 401},
        # the benchmark's inference batch
        {"name": "predict_65536", "kind": "predict", "queries": 65_536},
        # an epoch over 16384 scenarios (5 % held out) in batches of 2048
        {"name": "train_15564", "kind": "train", "rows": 15_564, "batch": 2048},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["trace", "trace", "trace", "build", "build", "sweep", "simulate", "predict", "predict", "train"])
    if kind == "trace":
        scene = rng.choice(["full", "full", "disc", "dense", "parity"])
        hi = {"full": 1e8, "disc": 3e7, "dense": 1e5, "parity": 3e5}[scene]
        lo = {"full": 1e5, "disc": 1e4, "dense": 5e3, "parity": 1e4}[scene]
        return {"kind": kind, "scene": scene, "photons": _log_int(rng, lo, hi)}
    if kind == "build":
        field = rng.choice(["grid", "meridional", "uniform", "uniform"])
        return {"kind": kind, "field": field, "bins": rng.randint(1, 64), "angles": rng.randint(257, 2401),
                "fast": field == "uniform" and rng.random() < 0.6, "max_um": math.exp(rng.uniform(math.log(5), math.log(300)))}
    if kind == "sweep":
        scenarios = _log_int(rng, 3, 256)
        return {"kind": kind, "scenarios": scenarios, "photons": _log_int(rng, 1e4, min(4e6, 1.28e8 / scenarios))}
    if kind == "simulate":
        return {"kind": kind, "material": rng.choice(["loess", "kaolin"]), "photons": _log_int(rng, 2e4, 1e6)}
    if kind == "predict":
        return {"kind": kind, "queries": _log_int(rng, 1, 410_624)}
    batch = 128 * rng.choice([2, 4, 8, 16, 24])
    return {"kind": kind, "rows": batch + _log_int(rng, 1, 20_000), "batch": batch}


# ---- inputs -----------------------------------------------------------------------------------------------
def _trace_scene(name):
    """(config, particles, sediment grid or None, grid top or None) of a traced scene."""
    if name == "full":
        return S.full_scene_workload()
    if name == "disc":
        return S.small_plain_workload()
    if name == "dense":
        core = 0.005
        cfg = S.small_cell_config(particle_surface_rms_slope_deg=0.0, wave_surface_rms_height_m=0.0,
                                  free_surface_model="rankine_vortex", vortex_core_radius_m=core,
                                  vortex_wall_center_height_difference_m=S.stirrer_rankine_delta_h(1200.0, core, 0.0125))
        cfg.validate()
        return cfg, S.kaolin_clay_particles(20_000.0), None, None
    cfg = S.small_cell_config()  # rough spheroids: the reference's default surfaces
    cfg.validate()
    return cfg, S.quartz_particles(concentration_mg_l=2000.0), None, None


def _population(case, rng):
    """A size distribution whose largest bin is case["max_um"], with a random median, width, index and amount."""
    top = float(case["max_um"])
    return S.quartz_particles(concentration_mg_l=float(np.exp(rng.uniform(0.0, np.log(1e3)))), n_bins=int(case["bins"]),
                              median_um=float(np.exp(rng.uniform(np.log(top / 60.0), np.log(top / 2.0)))),
                              sigma_g=float(rng.uniform(1.3, 2.0)), d_min_um=top / 200.0, d_max_um=top,
                              n=float(rng.uniform(1.50, 1.60)))


def _build_inputs(case, seed):
    rng = np.random.default_rng(int(seed))
    parts = _population(case, rng)
    over = dict(mie_phase_grid_size=int(case["angles"]))
    grid = zmax = None
    if case["field"] != "uniform":
        over.update(free_surface_model="localized_scully_vortex", vortex_core_radius_m=0.005,
                    vortex_wall_center_height_difference_m=float(rng.uniform(0.002, 0.008)),
                    sediment_transport_model="schiller_naumann_meridional_advection_diffusion")
    cfg = S.small_cell_config(**over)
    cfg.validate()
    if case["field"] == "grid":
        grid, zmax = S.rouse_radial_grid(cfg, parts.diameter_m.size, rouse=float(rng.uniform(0.1, 0.6)))
    return cfg, parts, grid, zmax


def _mlp_params(seed):
    """Weights and biases uniform in +-1/sqrt(fan in): W1 [256][6], b1, W2 [256][256], b2, W3, b3, W4, b4, W5 [3][256], b5."""
    rng = np.random.default_rng(int(seed) + 1)
    out = []
    for fan_in, units in ((6, 256), (256, 256), (256, 256), (256, 256), (256, 3)):
        b = 1.0 / math.sqrt(fan_in)
        out += [rng.uniform(-b, b, units * fan_in), rng.uniform(-b, b, units)]
    return np.concatenate(out).astype(np.float32)


def _mlp_rows(n, seed):
    """Standardised inputs and a smooth target of them with label noise."""
    rng = np.random.default_rng(int(seed) + 2)
    x = rng.normal(size=(n, 6)).astype(np.float32)
    t = np.stack([np.sin(x[:, 0]) + 0.5 * x[:, 1] * x[:, 2], np.cos(x[:, 3]) * x[:, 4], 0.3 * x[:, 5] ** 2 - x[:, 0]], 1)
    return x, (t + 0.05 * rng.normal(size=t.shape)).astype(np.float32)


def _epoch(case, seed):
    """Training rows (95 % of the data), in random order, cut to whole batches."""
    n, batch = int(case["rows"]), int(case["batch"])
    return np.random.default_rng(int(seed) + 3).permutation(n)[: n // batch * batch].astype(np.int32)


LEARNING_RATE = 1e-3  # the middle of the training's cosine schedule


def prepare(case, seed):
    kind = case["kind"]
    if kind == "trace":
        cfg, parts, grid, zmax = _trace_scene(case["scene"])
        ctx = L.Context(0)
        ctx.set_scene(cfg.to_scene_params())
        ctx.build_particles(parts.spec(cfg), cfg.sediment_spec(grid, zmax))
        weighted = case["scene"] == "dense"
        run_ = S.run_params(int(case["photons"]), seed=int(seed),
                            rng_mode=abi.RNG_REFERENCE_XORSHIFT if case["scene"] == "parity" else abi.RNG_PHILOX,
                            weight_mode=abi.WEIGHT_IMPLICIT if weighted else abi.WEIGHT_ANALOG)
        return {"kind": kind, "ctx": ctx, "run": run_, "records": case["scene"] == "parity"}
    if kind == "build":
        cfg, parts, grid, zmax = _build_inputs(case, seed)
        spec = parts.spec(cfg, table_arithmetic=abi.TABLES_FAST if case["fast"] else abi.TABLES_REFERENCE)
        return {"kind": kind, "ctx": L.Context(0), "scene": cfg.to_scene_params(), "particles": spec,
                "sediment": cfg.sediment_spec(grid, zmax), "solved": case["field"] == "meridional"}
    if kind == "sweep":
        n = int(case["photons"])
        scs = S.sweep_workload(int(case["scenarios"]), sampler_seed=int(seed), photons=(n, n))
        scenes, parts, seds = S.sweep_specs(scs, table_arithmetic=abi.TABLES_FAST)
        runs = [S.run_params(sc.n_photons, seed=sc.seed + int(seed), rng_mode=abi.RNG_PHILOX, scenario_id=i)
                for i, sc in enumerate(scs)]
        return {"kind": kind, "ctx": L.Context(0), "scenarios": scs, "scenes": scenes, "particles": parts,
                "sediments": seds, "runs": runs}
    if kind == "simulate":
        model = F.ClaritasForwardModel(particle_event_model="hybrid_mie_exact_rate")
        c = float(np.exp(np.random.default_rng(int(seed)).uniform(np.log(0.1), np.log(2.0))))
        return {"kind": kind, "model": model, "material": case["material"], "concentration": c,
                "photons": int(case["photons"]), "seed": int(seed)}
    if kind == "predict":
        model = G.Surrogate(0, max_batch=128, seed=0)
        model.net.set_params(_mlp_params(seed))
        x, _ = _mlp_rows(int(case["queries"]), seed)
        return {"kind": kind, "model": model, "x": torch.from_numpy(x).cuda()}
    net = L.Network(0, max_batch=int(case["batch"]), seed=0)
    net.set_params(_mlp_params(seed))
    x, t = _mlp_rows(int(case["rows"]), seed)
    return {"kind": kind, "net": net, "x": torch.from_numpy(x).cuda(), "t": torch.from_numpy(t).cuda(),
            "order": torch.from_numpy(_epoch(case, seed)), "batch": int(case["batch"])}


# ---- one pass ---------------------------------------------------------------------------------------------
def _tallies(t):
    """Every field of a tally set but the scheduler's own statistics (which queue was visited how often)."""
    return {k: v for k, v in t.items() if k not in ("sched_stats", "reserved")}


def run(state):
    kind = state["kind"]
    if kind == "trace":
        t, rec = state["ctx"].trace(state["run"], records=state["records"])
        out = _tallies(t)
        if rec is not None:  # the record columns: 27 whole numbers and 8 values per ray
            cols = rec.view(np.int32).reshape(rec.shape[0], -1)
            k = len(abi.RECORD_INT_FIELDS)
            out["record_counts"], out["record_values"] = cols[:, :k], cols[:, k:].view(np.float32)
        return out
    if kind == "build":
        ctx = state["ctx"]
        ctx.set_scene(state["scene"])
        ctx.build_particles(state["particles"], state["sediment"])
        out = ctx.physics()
        if state["solved"]:
            out.update(ctx.sediment_field())
        return out
    if kind == "sweep":
        ctx = state["ctx"]
        ctx.sweep_build(state["scenes"], state["particles"], state["sediments"])
        ts = [_tallies(t) for t in ctx.sweep_trace(state["runs"])]
        return {k: np.stack([t[k] for t in ts]) for k in ts[0]}
    if kind == "simulate":
        r = state["model"].simulate(state["material"], state["concentration"], n_rays=state["photons"], seed=state["seed"])
        return {k: v for k, v in vars(r).items() if isinstance(v, np.ndarray) and v.dtype.kind in "fiub"}
    if kind == "predict":
        return state["model"].predict_device(state["x"])
    idx = state["order"].cuda()  # an epoch's order is drawn on the host
    x, t, net = state["x"], state["t"], state["net"]
    loss = net.train(x.data_ptr(), t.data_ptr(), idx.data_ptr(), idx.numel(), state["batch"], LEARNING_RATE)
    return {"loss": loss, "params": net.get_params()}


# ---- what a pass cannot do without --------------------------------------------------------------------------
def _mie_orders(d, n_medium, wavelength):
    x = math.pi * n_medium * np.asarray(d) / wavelength
    return np.floor(x + 4.0 * np.cbrt(x) + 2.0).astype(int)


def work(case):
    kind = case["kind"]
    if kind == "trace":
        n = int(case["photons"])
        out = n * 35 * 4 if case["scene"] == "parity" else 0
        return {"bytes": 1e6 + out, "flops": n * OPS_PER_PHOTON[case["scene"]]}
    if kind == "build":
        cfg, parts, grid, _ = _build_inputs(case, 0)
        orders = float(_mie_orders(parts.diameter_m, cfg.n_water, cfg.particle_wavelength_m).sum())
        n, nt = int(case["bins"]), int(case["angles"])
        cells = 48 * 96 if case["field"] == "meridional" else (0 if grid is None else grid[0].size)
        # S1 and S2 of two mirrored angles: eight multiply-adds per order; 1250 relaxations of the solved field
        flops = orders * nt * 8.0 + orders * 200.0 + (n * cells * 12.0 * 1250 if case["field"] == "meridional" else 0.0)
        return {"bytes": 8.0 * (n * nt + nt + 24 * n + n * cells), "flops": flops}
    if kind == "sweep":
        n, m = int(case["scenarios"]), int(case["photons"])
        d = np.geomspace(1e-6, 200e-6, 64)
        orders = float(_mie_orders(d, 1.33, 860e-9).sum())
        return {"bytes": n * 64 * 1801 * 12.0, "flops": n * (orders * 1801 * 8.0 + m * OPS_PER_PHOTON["sweep"])}
    if kind == "simulate":
        return {"bytes": 1e6, "flops": int(case["photons"]) * OPS_PER_PHOTON["simulate"]}
    if kind == "predict":
        n = int(case["queries"])
        return {"bytes": n * 36.0 + MLP_PARAMS * 2.0, "flops": float(n) * MLP_FLOP}
    n = int(case["rows"]) // int(case["batch"]) * int(case["batch"])
    return {"bytes": n * 40.0 + n / int(case["batch"]) * MLP_PARAMS * 24.0, "flops": 3.0 * n * MLP_FLOP}


# ---- the values in 64 bits --------------------------------------------------------------------------------
def _mie_exact(d, m, n_medium, wavelength):
    """Bohren & Huffman's series of one sphere: (x, qext, qsca, qback, g, (a_n, b_n)).
    psi_n and the logarithmic derivative by downward recurrence, chi_n upward (each in its stable direction)."""
    x = math.pi * n_medium * d / wavelength
    stop = int(x + 4.0 * x ** (1.0 / 3.0) + 2.0)
    start = int(max(stop, abs(m * x))) + 200
    z = m * x
    D = np.zeros(start + 1, dtype=complex)
    for n in range(start, 0, -1):
        D[n - 1] = n / z - 1.0 / (D[n] + n / z)
    r = np.zeros(start + 2)  # psi_n / psi_{n-1}
    for n in range(start, 0, -1):
        r[n] = 1.0 / ((2 * n + 1) / x - r[n + 1])
    psi, chi = np.zeros(stop + 1), np.zeros(stop + 1)
    # psi_0 = sin x and psi_1 = sin x / x - cos x never vanish together: anchor on the larger one
    psi[0], psi[1] = math.sin(x), math.sin(x) / x - math.cos(x)
    if abs(psi[0]) >= abs(psi[1]):
        psi[1] = psi[0] * r[1]
    for n in range(2, stop + 1):
        psi[n] = psi[n - 1] * r[n]
    chi[0], chi[1] = math.cos(x), math.cos(x) / x + math.sin(x)
    for n in range(2, stop + 1):
        chi[n] = (2 * n - 1) / x * chi[n - 1] - chi[n - 2]
    n = np.arange(1, stop + 1)
    xi = psi - 1j * chi
    ca, cb = D[1:stop + 1] / m + n / x, m * D[1:stop + 1] + n / x
    a = (ca * psi[1:] - psi[:-1]) / (ca * xi[1:] - xi[:-1])
    b = (cb * psi[1:] - psi[:-1]) / (cb * xi[1:] - xi[:-1])
    qe = 2.0 / x ** 2 * np.sum((2 * n + 1) * (a + b).real)
    qs = 2.0 / x ** 2 * np.sum((2 * n + 1) * (abs(a) ** 2 + abs(b) ** 2))
    qb = abs(np.sum((2 * n + 1) * (-1.0) ** n * (a - b))) ** 2 / x ** 2
    t = np.sum((2 * n + 1) / (n * (n + 1.0)) * (a * b.conj()).real)
    t += np.sum((n * (n + 2.0) / (n + 1.0))[:-1] * (a[:-1] * a[1:].conj() + b[:-1] * b[1:].conj()).real)
    return x, qe, qs, qb, 4.0 * t / (x ** 2 * qs), (a, b)


def _tables_exact(cfg, parts, nt):
    u = np.arange(nt) / (nt - 1.0)
    theta = 0.5 * math.pi * (1.0 - np.cos(math.pi * u))
    theta[0], theta[-1] = 0.0, math.pi
    mu = np.cos(theta)
    rows = [_mie_exact(float(d), complex(nr, k) / cfg.n_water, cfg.n_water, cfg.particle_wavelength_m)
            for d, nr, k in zip(parts.diameter_m, parts.n_real, parts.k_imag)]
    top = max(r[5][0].size for r in rows)
    pi, tau = np.zeros((top + 1, nt)), np.zeros((top + 1, nt))
    pi[1] = 1.0
    for n in range(2, top + 1):
        pi[n] = (2 * n - 1) / (n - 1.0) * mu * pi[n - 1] - n / (n - 1.0) * pi[n - 2]
    for n in range(1, top + 1):
        tau[n] = n * mu * pi[n] - (n + 1.0) * pi[n - 1]
    out = {k: np.array([r[i] for r in rows]) for i, k in enumerate(("size_parameter", "qext", "qsca", "qback", "asym_g"))}
    cdf = np.zeros((len(rows), nt))
    for i, r in enumerate(rows):
        a, b = r[5]
        n = np.arange(1, a.size + 1)
        c = (2 * n + 1) / (n * (n + 1.0))
        s1 = (c * a) @ pi[1:a.size + 1] + (c * b) @ tau[1:a.size + 1]
        s2 = (c * a) @ tau[1:a.size + 1] + (c * b) @ pi[1:a.size + 1]
        pdf = 0.5 * (abs(s1) ** 2 + abs(s2) ** 2) * np.sin(theta)
        cum = np.concatenate([[0.0], np.cumsum(0.5 * (pdf[1:] + pdf[:-1]) * np.diff(theta))])
        cdf[i] = cum / cum[-1]
    out.update(theta=theta, phase_cdf=cdf)
    return out


def _mlp_tensors(params, device):
    p = torch.from_numpy(params.astype(np.float64)).to(device)
    w, at = [], 0
    for fan_in, units in ((6, 256), (256, 256), (256, 256), (256, 256), (256, 3)):
        w += [p[at:at + units * fan_in].reshape(units, fan_in).clone(), p[at + units * fan_in:at + units * (fan_in + 1)].clone()]
        at += units * (fan_in + 1)
    return w


def _mlp_forward(w, x):
    for k in range(4):
        x = torch.nn.functional.silu(x @ w[2 * k].T + w[2 * k + 1])
    return x @ w[8].T + w[9]


def exact(case, seed):
    kind = case["kind"]
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    if kind == "build":
        cfg, parts, _, _ = _build_inputs(case, seed)
        return _tables_exact(cfg, parts, int(case["angles"]))
    if kind == "predict":
        x = torch.from_numpy(_mlp_rows(int(case["queries"]), seed)[0].astype(np.float64)).to(dev)
        with torch.no_grad():
            return _mlp_forward(_mlp_tensors(_mlp_params(seed), dev), x)
    if kind == "train":
        w = [v.requires_grad_(True) for v in _mlp_tensors(_mlp_params(seed), dev)]
        x, t = (torch.from_numpy(v.astype(np.float64)).to(dev) for v in _mlp_rows(int(case["rows"]), seed))
        order = torch.from_numpy(_epoch(case, seed).astype(np.int64)).to(dev).reshape(-1, int(case["batch"]))
        adam = torch.optim.Adam(w, lr=LEARNING_RATE)
        total = 0.0
        for idx in order:
            loss = ((_mlp_forward(w, x[idx]) - t[idx]) ** 2).mean()
            adam.zero_grad()
            loss.backward()
            adam.step()
            total += float(loss.detach())
        return {"loss": total / len(order), "params": torch.cat([v.detach().reshape(-1) for v in w]).cpu().numpy()}
    return None
