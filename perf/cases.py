"""The framework's workloads as timed cases: check intervals of REWL batches (2D Ising and 2D
Ashkin-Teller, with and without per-bin observables), the warm-start network (prediction, one
gradient, training steps) and the canonical thermodynamics of a converged run.

A case is a dict with a "kind":
  ising / at / mixed   restore a checkpoint, run one check interval, write the checkpoint back: the
                       state a job scheduler keeps on the host between intervals.  With observables
                       the pass ends with the per-window averages instead, as a run's end does.
  predict              MLP.predict on the bins of a lattice's windows (host rows in, host values out)
  gradient             forward + backward of one batch, gradients read back
  train                Adam steps on a training set held by the network, weights read back
  thermo               the temperature ladder of a density of states
"""
from __future__ import annotations

import math

import numpy as np
import torch

import rewl_simulator_gb300 as rg
from rewl_simulator_gb300.mlp import MLP
from rewl_simulator_gb300.thermo import thermodynamics


def _ising(L, windows, replicas, se, sc, **kw):
    return dict(kind="ising", L=L, windows=windows, replicas=replicas, sweeps_per_exchange=se, sweeps_per_check=sc,
                observables=0, one_over_t=0, stage=0, graphs=1, **kw)


def _at(L, windows, replicas, real, se, sc, **kw):
    return dict(kind="at", L=L, windows=windows, replicas=replicas, realisations=real, sweeps_per_exchange=se,
                sweeps_per_check=sc, observables=0, K=0.5, sigma_h=0.5, bin_width=0.05, graphs=0, **kw)


def listed():
    return [
        # a smoke-sized run: launches, synchronisations and the host loop weigh as much as the sweeps
        dict(_ising(8, 3, 2, 20, 40), name="ising_L8_3x2", graphs=0),
        # the reference's default build: 1/t schedule, moments and correlation lengths per bin
        dict(_ising(16, 16, 4, 100, 200), name="ising_L16_16x4_corr", observables=2, one_over_t=1),
        # a lattice whose rows are no power of two (chunks of 20 sites), fresh tables
        dict(_ising(20, 8, 4, 100, 200), name="ising_L20_8x4"),
        # batched Ising L = 32, 16 windows x 8 walkers, late stage (ln f ~ 1e-5, converged tables)
        dict(_ising(32, 16, 8, 500, 1000), name="ising_L32_16x8", stage=17),
        # the headline configuration: Ising L = 64, 64 windows x 8 walkers, 1/t schedule
        dict(_ising(64, 64, 8, 250, 500), name="ising_L64_64x8", stage=17, one_over_t=1),
        # the same lattice with 48 walkers per window: a device full of walkers
        dict(_ising(64, 64, 48, 125, 250), name="ising_L64_64x48", stage=17, one_over_t=1),
        # Ashkin-Teller with Baxter fields and all observables, a small lattice
        dict(_at(12, 4, 4, 2, 100, 200), name="at_L12_4x4_corr", observables=2),
        # Ashkin-Teller L = 32, 16 disorder realisations x 8 windows x 4 walkers
        dict(_at(32, 8, 4, 16, 100, 200), name="at_L32_16real"),
        # an uneven batch: Ising L = 16, 24, 32 and Ashkin-Teller L = 24 in one engine
        dict(kind="mixed", name="mixed_ising_at", L_ising=16, L_ising2=24, L_ising3=32, L_at=24, realisations=4,
             windows=8, replicas=4, sweeps_per_exchange=50, sweeps_per_check=100, graphs=1),
        # the warm start of an L = 64 instance: one prediction over the bins of all its windows
        dict(kind="predict", name="mlp_predict_7900", rows=7900, hidden=256, layers=4),
        # training as the warm start does it: batches of 4096 rows, Adam on FP32 masters
        dict(kind="train", name="mlp_train_b4096", rows=6012, batch=4096, steps=32, hidden=256, layers=4),
        # the reference's default ladder (50,000 temperatures) over an L = 64 density of states
        dict(kind="thermo", name="thermo_4095x50000", levels=4095, L=64, temperatures=50000, obs=5, trapezoid=True),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["ising", "ising", "ising", "at", "at", "mixed", "predict", "gradient", "train", "thermo"])
    if kind == "ising":
        L = rng.choice([_log_int(rng, 6, 64), 8 * rng.randint(1, 8)])
        windows = max(1, min(_log_int(rng, 2, 64), L * L // 16))
        replicas = _log_int(rng, 1, 48)
        sweeps = max(4, min(_log_int(rng, 20, 400), 500_000 // (L * L)))
        c = _ising(L, windows, replicas, sweeps, sweeps * rng.choice([1, 2]))
        c["observables"] = rng.choice([0, 0, 0, 1, 2])
        if c["observables"]:
            c["windows"], c["replicas"] = min(windows, 16), min(replicas, 8)
        c["one_over_t"] = rng.choice([0, 1])
        c["stage"] = rng.choice([0, 8, 17])
        c["graphs"] = rng.choice([0, 1])
        return c
    if kind == "at":
        L = _log_int(rng, 5, 32)
        real = max(1, min(_log_int(rng, 1, 16), 16 * 1024 // (L * L)))
        sweeps = max(4, min(_log_int(rng, 10, 100), 100_000 // (L * L)))
        c = _at(L, rng.randint(2, 8), rng.randint(1, 4), real, sweeps, sweeps * rng.choice([1, 2]))
        c["observables"] = rng.choice([0, 0, 1, 2])
        c["K"] = rng.choice([0.0, 0.25, 0.5, 0.75])
        c["sigma_h"] = rng.choice([0.0, 0.3, 0.5])
        c["bin_width"] = rng.choice([0.05, 0.05, 0.25, 1.0])
        if c["observables"]:
            c["realisations"] = 1
        return c
    if kind == "mixed":
        return dict(kind="mixed", L_ising=rng.randint(6, 16), L_ising2=4 * rng.randint(4, 8), L_ising3=rng.randint(17, 32),
                    L_at=rng.randint(6, 24), realisations=rng.randint(1, 4), windows=rng.randint(2, 8),
                    replicas=rng.randint(1, 4), sweeps_per_exchange=_log_int(rng, 10, 50), sweeps_per_check=0,
                    graphs=rng.choice([0, 1]))
    hidden, layers = rng.choice([64, 128, 256, 256, 256]), rng.randint(2, 5)
    if kind == "predict":
        return dict(kind="predict", rows=_log_int(rng, 30, 16000), hidden=hidden, layers=layers)
    if kind == "gradient":
        return dict(kind="gradient", rows=64 * _log_int(rng, 1, 64), hidden=hidden, layers=layers)
    if kind == "train":
        return dict(kind="train", rows=_log_int(rng, 300, 10000), batch=64 * _log_int(rng, 2, 64),
                    steps=_log_int(rng, 4, 32), hidden=hidden, layers=layers)
    L = _log_int(rng, 6, 64)
    return dict(kind="thermo", levels=max(20, min(4095, L * L - rng.randint(0, 5))), L=L,
                temperatures=_log_int(rng, 500, 50000), obs=rng.choice([0, 0, 4, 5, 13, 17]),
                trapezoid=rng.choice([True, False]))


# ---------------------------------------------------------------------------------------------
# REWL check intervals
# ---------------------------------------------------------------------------------------------
def _ising_span(L):
    """Energy range of an L x L torus that single flips reach: the whole spectrum for even L, its
    lower half for odd L (whose antiferromagnetic top is frustrated)."""
    N = L * L
    return (-2.0 * N, 2.0 * N + 4) if L % 2 == 0 else (-2.0 * N, -2.0 * N + 4.0 * (N // 2))


def _ising_instance(L, windows, replicas, seed):
    lo, hi = _ising_span(L)
    return rg.Instance(model=rg.MODEL_ISING2D, L=L, energy_min=lo, energy_max=hi, bin_width=4.0, num_windows=windows,
                       replicas_per_window=replicas, window_overlap=0.75, init_mode=0, seed=seed)


def _at_instance(L, K, sigma_h, bin_width, windows, replicas, seed):
    N = L * L
    h = None
    if sigma_h > 0:
        h = np.round(np.random.default_rng(seed).normal(0.0, sigma_h, N) * 2**20) / 2**20
    return rg.Instance(model=rg.MODEL_ASHKIN_TELLER2D, L=L, K=K, fields=h, energy_min=-math.ceil((2.0 + K) * 2) * float(N),
                       energy_max=0.0, bin_width=bin_width, num_windows=windows, replicas_per_window=replicas,
                       window_overlap=0.75, seed=seed)


def _onsager_entropy(L):
    """Entropy per site of the 2D Ising model as a function of the energy per site (J = 1), from
    Onsager's free energy with the integrals as sums over the L x L midpoint grid."""
    beta = np.concatenate([np.linspace(0.0, 0.7, 281), np.linspace(0.71, 3.0, 230)])
    k = (np.arange(max(L, 32)) + 0.5) * math.pi / max(L, 32)
    cc = (np.cos(k)[:, None] + np.cos(k)[None, :]).reshape(-1)
    f = np.array([math.log(2.0) + 0.5 * np.mean(np.log(np.cosh(2 * b) ** 2 - np.sinh(2 * b) * cc)) for b in beta])
    u = -np.gradient(f, beta)
    s = f + beta * u
    order = np.argsort(u)
    return lambda e: np.interp(-np.abs(e), u[order], np.maximum(s[order], 0.0))


def _instances(case, seed):
    base = 1_000_003 * (seed + 1)
    w, r = case["windows"], case["replicas"]
    if case["kind"] == "ising":
        return [_ising_instance(case["L"], w, r, base)]
    if case["kind"] == "at":
        return [_at_instance(case["L"], case["K"], case["sigma_h"], case["bin_width"], w, r, base + 7 * k)
                for k in range(case["realisations"])]
    inss = [_ising_instance(case[k], min(w, case[k] ** 2 // 16), r, base + i)
            for i, k in enumerate(("L_ising", "L_ising2", "L_ising3"))]
    return inss + [_at_instance(case["L_at"], K, 0.3, 0.05, w, r, base + 100 + 7 * k)
                   for k in range(case["realisations"]) for K in (0.25, 0.5)]


def _prepare_engine(case, seed):
    inss = _instances(case, seed)
    at = case["kind"] != "ising"
    se = case["sweeps_per_exchange"]
    batch = rg.Batch(instances=inss, sweeps_per_exchange=se, sweeps_per_check=case["sweeps_per_check"] or se,
                     flatness_param=0.8, lnf_initial=1.0, lnf_final=1e-8, one_over_t=case.get("one_over_t", 0),
                     mask_mode=rg.MASK_VISITED if at else rg.MASK_STATIC, observables=case.get("observables", 0),
                     graphs=case["graphs"])
    eng = rg.Engine(batch)
    stage = case.get("stage", 0)
    if stage:
        # a late stage: converged tables (to the accuracy of Onsager's free energy) and ln f = 2^-stage
        N = case["L"] ** 2
        s = _onsager_entropy(case["L"])
        for w, (lo, hi, nb) in enumerate(eng.windows[0]):
            g = N * s((lo + 4.0 * np.arange(nb)) / N)
            eng.set_logdos(0, w, g - g[0])
            eng.set_lnf(0, w, 2.0 ** -stage)
    eng.wang_landau_walk(se)              # leave the start configurations
    eng.replica_exchange_update()
    eng.check_flat()
    n = eng.snapshot_size()
    start = torch.empty(n, dtype=torch.uint8, pin_memory=True).zero_()
    end = torch.empty(n, dtype=torch.uint8, pin_memory=True).zero_()
    eng.snapshot_into(start.data_ptr(), n)
    return dict(kind="engine", eng=eng, start=start, end=end, n=n, observables=batch.observables)


def _run_engine(st):
    eng = st["eng"]
    eng.restore_from(st["start"].data_ptr(), st["n"])
    status = eng.run_cycles(1)
    out = dict(status=np.array([status.sweeps, status.cycles, status.flat_events, status.windows_done,
                                status.exchanges_attempted, status.exchanges_accepted, status.attempted_flips]))
    if st["observables"]:
        pairs = [(i, w) for i, ws in enumerate(eng.windows) for w in range(len(ws))]
        out["observables"] = np.concatenate([eng.window_observables(i, w).reshape(-1) for i, w in pairs])
        out["logdos"] = np.concatenate([eng.window_logdos(i, w) for i, w in pairs])
    else:
        eng.snapshot_into(st["end"].data_ptr(), st["n"])
        out["state"] = st["end"]
    return out


def _engine_work(case):
    """Attempted flips (a dozen integer operations each at least: two neighbour sums, the uniform,
    the comparison, the update) and the checkpoint read and written."""
    flips = state = 0
    for ins in _instances(case, 0):
        walkers = ins.num_windows * ins.replicas_per_window
        flips += walkers * ins.ndof * (case["sweeps_per_check"] or case["sweeps_per_exchange"])
        bins = (ins.energy_max - ins.energy_min) / ins.bin_width / (1 + 0.25 * (ins.num_windows - 1))
        state += walkers * (ins.ndof + 20 * bins)
    return {"bytes": 2.0 * state, "flops": 24.0 * flips}


# ---------------------------------------------------------------------------------------------
# Warm-start network
# ---------------------------------------------------------------------------------------------
_PAD_IN, _PAD_OUT, _IN = 64, 64, 7


def _layout(hidden, layers):
    """(input width, output width, weight offset, bias offset) per layer of the padded parameters."""
    rows, off = [], 0
    for l in range(layers + 1):
        din, dout = _PAD_IN if l == 0 else hidden, _PAD_OUT if l == layers else hidden
        rows.append((din, dout, off, off + din * dout))
        off = (off + din * dout + dout + 7) // 8 * 8
    return rows, off


def _mlp_inputs(case, seed):
    """Rows of the features the warm start uses, targets shaped like ln g/N, and weights at the
    usual uniform(+-1/sqrt(fan-in)) scale."""
    r = np.random.default_rng(seed)
    n = case["rows"]
    X = np.empty((n, _IN), dtype=np.float32)
    X[:, 0] = r.uniform(-2.0, 2.0, n)
    X[:, 1] = 1.0 / r.choice([16, 24, 32, 64], n)
    X[:, 2] = 1.0
    X[:, 3] = r.choice([0.0, 0.5], n)
    X[:, 4] = r.choice([0.0, 0.5], n)
    X[:, 5] = np.floor(X[:, 0] * 8) / 8
    X[:, 6] = X[:, 5] + 0.25
    y = (math.log(2.0) - 0.25 * X[:, 0] ** 2 + 0.3 * X[:, 1] * np.cos(3 * X[:, 0])).astype(np.float32)
    rows, size = _layout(case["hidden"], case["layers"])
    p = np.zeros(size, dtype=np.float32)
    for l, (din, dout, wo, bo) in enumerate(rows):
        i, o = (_IN if l == 0 else din), (1 if l == case["layers"] else dout)
        b = 1.0 / math.sqrt(i)
        w = np.zeros((dout, din), dtype=np.float32)
        w[:o, :i] = r.uniform(-b, b, (o, i))
        p[wo:wo + dout * din] = w.reshape(-1)
        p[bo:bo + o] = r.uniform(-b, b, o)
    return X, y, p


def _prepare_mlp(case, seed):
    X, y, p = _mlp_inputs(case, seed)
    m = MLP(hidden=case["hidden"], layers=case["layers"], seed=seed + 1)
    m.set_params(p)
    if case["kind"] == "train":
        m.set_data(X, y)
    return dict(kind=case["kind"], mlp=m, X=X, y=y, steps=case.get("steps"), batch=case.get("batch"))


def _run_mlp(st):
    m = st["mlp"]
    if st["kind"] == "predict":
        return dict(y=m.predict(st["X"]))
    if st["kind"] == "gradient":
        return dict(loss=m.gradient(st["X"], st["y"]), grads=m.grads())
    losses = m.train(st["steps"], batch=st["batch"], lr=1e-3)
    return dict(losses=losses, params=m.params())


def _mlp_work(case):
    h, n = case["hidden"], case["layers"]
    macs = _IN * h + (n - 1) * h * h + h
    params = macs + n * h + 1
    if case["kind"] == "predict":
        return {"bytes": 4.0 * case["rows"] * (_IN + 1) + 4.0 * params, "flops": 2.0 * macs * case["rows"]}
    if case["kind"] == "gradient":
        return {"bytes": 4.0 * case["rows"] * (_IN + 1) + 8.0 * params, "flops": 6.0 * macs * case["rows"]}
    rows = case["batch"] * case["steps"]
    # per step the batch and, for Adam, weights and both moments read and written
    return {"bytes": 4.0 * rows * (_IN + 1) + 24.0 * params * case["steps"], "flops": 6.0 * macs * rows}


def _exact_mlp(case, seed):
    """The network in 64 bits.  A training trajectory has no value to compare with: its batches are
    the network's own draws."""
    if case["kind"] == "train":
        return None
    X, y, p = _mlp_inputs(case, seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    p64 = torch.tensor(p, dtype=torch.float64, device=dev, requires_grad=case["kind"] == "gradient")
    rows, _ = _layout(case["hidden"], case["layers"])
    a = torch.zeros((len(X), _PAD_IN), dtype=torch.float64, device=dev)
    a[:, :_IN] = torch.tensor(X, dtype=torch.float64, device=dev)
    for l, (din, dout, wo, bo) in enumerate(rows):
        a = a @ p64[wo:wo + din * dout].reshape(dout, din).T + p64[bo:bo + dout]
        if l < case["layers"]:
            a = torch.nn.functional.gelu(a)
    if case["kind"] == "predict":
        return dict(y=a[:, 0].cpu().numpy())
    loss = ((a[:, 0] - torch.tensor(y, dtype=torch.float64, device=dev)) ** 2).mean()
    loss.backward()
    g = p64.grad
    # entries of the padding are no parameters: their gradient is reported as computed from the
    # padded inputs and outputs, which are zero
    return dict(loss=float(loss.detach()), grads=g.cpu().numpy())


# ---------------------------------------------------------------------------------------------
# Thermodynamics
# ---------------------------------------------------------------------------------------------
def _thermo_inputs(case, seed):
    """A density of states on evenly spaced levels with the two unreachable ones left out, small
    Monte Carlo noise on it, and observable columns (moments, the last one a count)."""
    r = np.random.default_rng(seed)
    N, nb = case["L"] ** 2, case["levels"]
    k = np.arange(nb + 2)
    k = np.delete(k, [1, nb])
    e = -2.0 + 4.0 * k / (nb + 1)
    lng = N * _onsager_entropy(case["L"])(e)
    lng = lng - lng[0] + math.log(2.0) + r.normal(0.0, 0.02, nb)
    obs = None
    if case["obs"]:
        m = np.clip(np.abs(e) / 2 + r.normal(0, 0.01, nb), 1e-3, 1.0)
        obs = np.stack([m ** (1 + j % 4) for j in range(case["obs"])], axis=1)
        obs[:, -1] = r.integers(1000, 100000, nb)
    return e * N, lng, obs, N


def _prepare_thermo(case, seed):
    E, lng, obs, N = _thermo_inputs(case, seed)
    return dict(kind="thermo", E=E, lng=lng, obs=obs, N=N, num_T=case["temperatures"], trapezoid=case["trapezoid"])


def _run_thermo(st):
    obs = st["obs"]
    T, rows = thermodynamics(st["E"], st["lng"], st["N"], obs=obs, counts_col=-1 if obs is None else obs.shape[1] - 1,
                             num_T=st["num_T"], trapezoid=st["trapezoid"])
    return dict(T=T, free_energy=rows[:, 0], energy=rows[:, 1], energy2=rows[:, 2], entropy=rows[:, 3],
                heat=rows[:, 4], observables=rows[:, 5:])


def _exact_thermo(case, seed):
    E, lng, obs, N = _thermo_inputs(case, seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    Et, gt = (torch.tensor(v, dtype=torch.float64, device=dev) for v in (E, lng))
    half = torch.ones_like(Et)
    if case["trapezoid"]:
        half[0] = half[-1] = 0.5
    nT = case["temperatures"]
    T = torch.tensor(0.01 + (50.01 - 0.01) / nT * np.arange(nT), dtype=torch.float64, device=dev)
    cols = torch.tensor(obs[:, :-1], dtype=torch.float64, device=dev) if obs is not None else None
    out = {k: [] for k in ("free_energy", "energy", "energy2", "entropy", "heat", "observables")}
    for t in T.split(2048):
        x = gt[None, :] - Et[None, :] / t[:, None]
        m = x.max(dim=1, keepdim=True).values
        w = torch.exp(x - m) * half
        Z = w.sum(dim=1)
        p = w / Z[:, None]
        U, U2 = p @ Et / N, p @ (Et * Et) / N**2
        out["free_energy"].append(-t * (m[:, 0] + torch.log(Z)) / N)
        out["energy"].append(U)
        out["energy2"].append(U2)
        out["entropy"].append(p @ gt / N)
        # the variance around the mean: the same number as U2 - U^2 without its cancellation
        out["heat"].append((p * (Et[None, :] - N * U[:, None]) ** 2).sum(dim=1) / (N * t * t))
        if cols is not None:
            mean = torch.full((len(t), 1), float(obs[:, -1].mean()), dtype=torch.float64, device=dev)
            out["observables"].append(torch.cat([p @ cols, mean], dim=1))
        else:
            out["observables"].append(torch.zeros((len(t), 0), dtype=torch.float64, device=dev))
    return dict(T=T.cpu().numpy(), **{k: torch.cat(v).cpu().numpy() for k, v in out.items()})


def _thermo_work(case):
    """Per temperature and level: the exponent (2), its exponential (counted 10), five sums and the
    observables' (2 each), in FP64."""
    pairs = float(case["levels"]) * case["temperatures"]
    return {"bytes": 8.0 * case["levels"] * (2 + case["obs"]) + 8.0 * case["temperatures"] * (6 + case["obs"]),
            "flops": pairs * (22 + 2 * case["obs"])}


# ---------------------------------------------------------------------------------------------
def prepare(case, seed):
    if case["kind"] in ("ising", "at", "mixed"):
        return _prepare_engine(case, seed)
    if case["kind"] == "thermo":
        return _prepare_thermo(case, seed)
    return _prepare_mlp(case, seed)


def run(state):
    if state["kind"] == "engine":
        return _run_engine(state)
    if state["kind"] == "thermo":
        return _run_thermo(state)
    return _run_mlp(state)


def work(case):
    if case["kind"] in ("ising", "at", "mixed"):
        return _engine_work(case)
    if case["kind"] == "thermo":
        return _thermo_work(case)
    return _mlp_work(case)


def exact(case, seed):
    if case["kind"] == "thermo":
        return _exact_thermo(case, seed)
    if case["kind"] in ("predict", "gradient", "train"):
        return _exact_mlp(case, seed)
    return None           # whole numbers: lattices, tables, counters
