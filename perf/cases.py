"""What a user of the package has it do, as cases that can be timed and compared.

A case is a dict of plain values whose ``kind`` names the public call:

* ``simulate``   ``Simulator(model).simulate`` on host parameters, host arrays back
* ``predictive`` HSSM's ``rng_fn`` over one draw per data trial, host arrays back
* ``batch``      ``BatchedSimulator.run``: uneven sample counts per parameter set, on the device
* ``sets``       ``SetBatch.run``: equal sample counts for every simulator family, on the device
* ``records``    ``BatchedKdePipeline.run_batch``: simulate, fit, resample, evaluate, training records
* ``kde``        ``KdeBatch`` fit and ``evaluate`` on simulated data that is already there
* ``surrogate``  ``MlpSurrogate.forward`` on query rows
* ``gradient``   ``MlpSurrogate.loglik`` and its gradient with respect to theta
* ``train``      ``MlpSurrogate.train_step`` on a batch of records, mid-training

Parameters are drawn uniformly from each model's configured ``param_bounds``,
as the data generator draws them.  Every input is made from the seed alone.
"""

from __future__ import annotations

import math
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path.cwd() / "ssm-simulators_b200"))

from ssms_b200 import hssm_support  # noqa: E402
from ssms_b200.batch import BatchedSimulator  # noqa: E402
from ssms_b200.batch_models import SetBatch  # noqa: E402
from ssms_b200.config import model_config  # noqa: E402
from ssms_b200.dataset_generators import BatchedKdePipeline, get_lan_kde_config  # noqa: E402
from ssms_b200.kde import KdeBatch  # noqa: E402
from ssms_b200.simulator import Simulator  # noqa: E402
from ssms_b200.surrogate import MlpSurrogate  # noqa: E402

MAX_T, DT = 20.0, 0.001

#: Euler steps of an average walk over each model's parameter box (accumulators
#: are counted in ``ACCUMULATORS``), for ``work``.
STEPS = {"ddm": 840, "angle": 675, "weibull": 600, "full_ddm": 620, "ornstein": 1050, "levy": 1000,
         "conflict_ds": 990, "race_no_bias_angle_4": 440, "lca_no_bias_4": 820, "racing_diffusion_3": 611}
ACCUMULATORS = {"race_no_bias_angle_4": 4, "lca_no_bias_4": 4, "racing_diffusion_3": 3}
#: operations per accumulator-step: a Gaussian increment (12) and the update with its tests (4)
STEP_FLOPS = 16


def listed():
    return [
        # one parameter vector at the API's default sample count: a user's first call, all latency
        {"name": "simulate_ddm_1000", "kind": "simulate", "model": "ddm", "trials": 1, "samples": 1000},
        # one parameter vector, 1e5 samples: a smooth histogram or one KDE likelihood
        {"name": "simulate_ddm_100000", "kind": "simulate", "model": "ddm", "trials": 1, "samples": 100_000},
        # posterior predictive of one subject's session through HSSM: a draw per data trial
        {"name": "predictive_angle_500", "kind": "predictive", "model": "angle", "trials": 500},
        # the batched workload: thousands of parameter vectors with uneven sample counts in one launch
        {"name": "batch_angle_4096", "kind": "batch", "model": "angle", "sets": 4096, "lo": 1000, "hi": 20_000},
        # time-varying drift (conflict task), drift tables on the device
        {"name": "sets_conflict_ds_512", "kind": "sets", "model": "conflict_ds", "sets": 512, "samples": 10_000},
        # alpha-stable noise, another sampler than the Gaussian models'
        {"name": "sets_levy_509", "kind": "sets", "model": "levy", "sets": 509, "samples": 9973},
        # several accumulators per walk
        {"name": "sets_lca_1024", "kind": "sets", "model": "lca_no_bias_4", "sets": 1024, "samples": 10_000},
        # network training data: simulation, KDE, resampling, records and auxiliary labels
        {"name": "records_angle_256", "kind": "records", "model": "angle", "sets": 256, "samples": 50_000},
        # KDE likelihoods of data that was simulated before
        {"name": "kde_128x20000", "kind": "kde", "sets": 128, "points": 20_000, "queries": 1000},
        # likelihoods of a large set of observations under the network
        {"name": "surrogate_1000000", "kind": "surrogate", "rows": 1_000_000},
        # likelihoods and theta-gradients as a gradient-based sampler asks for them
        {"name": "gradient_100000", "kind": "gradient", "rows": 100_000},
        # one optimiser step of the network's training
        {"name": "train_8192", "kind": "train", "rows": 8192},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["simulate", "predictive", "batch", "sets", "sets", "records", "kde", "surrogate", "gradient",
                       "train"])
    if kind == "simulate":
        model = rng.choice(["ddm", "angle", "weibull", "full_ddm", "levy", "race_no_bias_angle_4"])
        trials = rng.choice([1, 1, _log_int(rng, 2, 64)])
        return {"kind": kind, "model": model, "trials": trials, "samples": _log_int(rng, 500, 200_000 // trials)}
    if kind == "predictive":
        model = rng.choice(["ddm", "angle", "weibull", "full_ddm"])
        return {"kind": kind, "model": model, "trials": _log_int(rng, 50, 5000)}
    if kind == "batch":
        model = rng.choice(["ddm", "angle", "weibull", "ornstein", "full_ddm"])
        lo = _log_int(rng, 200, 2000)
        return {"kind": kind, "model": model, "sets": _log_int(rng, 16, 2048), "lo": lo, "hi": lo * rng.randint(2, 8)}
    if kind == "sets":
        model = rng.choice(["conflict_ds", "levy", "race_no_bias_angle_4", "lca_no_bias_4", "racing_diffusion_3",
                            "full_ddm"])
        return {"kind": kind, "model": model, "sets": _log_int(rng, 16, 700), "samples": _log_int(rng, 500, 10_000)}
    if kind == "records":
        return {"kind": kind, "model": rng.choice(["angle", "ddm", "weibull"]), "sets": _log_int(rng, 32, 256),
                "samples": _log_int(rng, 1000, 50_000)}
    if kind == "kde":
        return {"kind": kind, "sets": _log_int(rng, 4, 200), "points": _log_int(rng, 1000, 20_000),
                "queries": _log_int(rng, 100, 1000)}
    if kind == "train":
        return {"kind": kind, "rows": _log_int(rng, 1000, 20_000)}
    return {"kind": kind, "rows": _log_int(rng, 1000, 1_000_000)}


# ---------------------------------------------------------------- inputs
def _theta(model, n, rng):
    """n parameter vectors, uniform in the model's box, as float32 host arrays."""
    cfg = model_config[model]
    lo, hi = cfg["param_bounds"]
    return {p: rng.uniform(a, b, n).astype(np.float32) for p, a, b in zip(cfg["params"], lo, hi)}


def _query_rows(n, rng):
    """theta, rt ~ U(0, 20), choice of the angle model, [n, 7] float32."""
    th = _theta("angle", n, rng)
    return np.stack([*(th[p] for p in model_config["angle"]["params"]),
                     rng.uniform(0.0, MAX_T, n).astype(np.float32),
                     rng.choice(np.asarray([-1.0, 1.0], np.float32), n)], axis=1)


def _network(seed):
    return MlpSurrogate("angle", seed=seed)


def _training_inputs(case, seed):
    """The batch of records and the optimiser's moments of a network in mid-training."""
    rng = np.random.default_rng([seed, 7])
    n = case["rows"]
    x = _query_rows(n, rng)
    y = -1.5 * np.abs(x[:, 5] - x[:, 3] - 1.0) - 1.0 + 0.3 * rng.standard_normal(n)
    rec = np.concatenate([x, np.maximum(y, -16.0).astype(np.float32)[:, None]], axis=1)
    n_par = 23141
    m = (0.02 * rng.standard_normal(n_par)).astype(np.float32)
    v = (0.02 * (0.2 + rng.random(n_par))).astype(np.float32) ** 2
    return rec, m, v


def _kde_inputs(case, seed):
    """Simulated data as a simulator leaves it on the device (rt float32 with
    a few omissions, choice +-1), and queries sorted by (set, choice)."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    S, N, Q = case["sets"], case["points"], case["queries"]
    uni = lambda *n: torch.rand(*n, generator=g, device="cuda")  # noqa: E731
    t0, a, pu = 0.1 + 1.5 * uni(S, 1), 0.3 + 1.2 * uni(S, 1), 0.1 + 0.8 * uni(S, 1)
    # rt of a diffusion with drift towards one bound: inverse-Gaussian draws
    # (Michael, Schucany & Haas) of mean a and shape a^2, truncated at 20 s
    y = torch.randn(S, N, generator=g, device="cuda") ** 2
    x = a + 0.5 * y - 0.5 * torch.sqrt(4.0 * a * y + y * y)
    dec = torch.where(uni(S, N) * (a + x) <= a, x, a * a / x)
    rts = (t0 + dec).clamp(max=MAX_T).float()
    rts = torch.where(uni(S, N) < 0.002, torch.full_like(rts, -999.0), rts)
    choices = torch.where(uni(S, N) < pu, 1, -1).to(torch.int32)
    n_up = (pu.reshape(-1) * Q).round().long().clamp(1, Q - 1).cpu().numpy()
    counts = np.stack([Q - n_up, n_up], axis=1).reshape(-1)
    qoff = np.concatenate([[0], np.cumsum(counts)]).astype(np.int64)
    q = 0.05 + 6.0 * uni(S * Q).double() ** 2
    soff = np.arange(S + 1, dtype=np.int64) * N
    return rts.reshape(-1).contiguous(), choices.reshape(-1).contiguous(), soff, qoff, q


def prepare(case, seed):
    kind = case["kind"]
    rng = np.random.default_rng(seed)
    st = {"kind": kind, "seed": int(seed) % (2**31 - 1)}
    if kind == "simulate":
        st["sim"], st["n"] = Simulator(case["model"]), case["samples"]
        if case["trials"] == 1 and case["model"] == "ddm":
            # a typical subject: v 1, a 1.5, z 0.5, t 0.2, give or take
            st["theta"] = {"v": rng.uniform(0.9, 1.1), "a": rng.uniform(1.4, 1.6), "z": 0.5, "t": 0.2}
        else:
            st["theta"] = _theta(case["model"], case["trials"], rng)
    elif kind == "predictive":
        th = _theta(case["model"], case["trials"], rng)
        st["args"] = [th[p] for p in model_config[case["model"]]["params"]]
        st["fun"] = hssm_support.get_simulator_fun_internal(case["model"])
    elif kind == "batch":
        th = _theta(case["model"], case["sets"], rng)
        # counts spread evenly over [lo, hi], dealt to the sets at random
        ns = rng.permutation(np.linspace(case["lo"], case["hi"], case["sets"]).round().astype(np.int64))
        st["sim"] = BatchedSimulator(case["model"], th, ns, max_t=MAX_T, delta_t=DT, seed=st["seed"])
    elif kind == "sets":
        sim = Simulator(case["model"])
        th = _theta(case["model"], case["sets"], rng)
        p = sim.prepare(th, n_samples=case["samples"], delta_t=DT, max_t=MAX_T, random_state=st["seed"])
        st["sets"] = SetBatch(model_config[case["model"]]["simulator"].__name__, p["theta"], p["boundary"],
                              case["samples"], max_t=MAX_T, delta_t=DT, drift=p["drift"])
    elif kind == "records":
        cfg = get_lan_kde_config(case["model"])
        cfg["simulator"]["n_samples"] = case["samples"]
        st["pipe"] = BatchedKdePipeline(cfg, model_config[case["model"]], batch_size=case["sets"])
        # not the pipeline's own sampler: its parameter order, and with it the
        # draws for one seed, differ between processes
        st["theta"] = _theta(case["model"], case["sets"], rng)
    elif kind == "kde":
        st["rts"], st["choices"], st["soff"], st["qoff"], st["q"] = _kde_inputs(case, seed)
    elif kind == "surrogate":
        st["net"] = _network(st["seed"])
        st["x"] = torch.from_numpy(_query_rows(case["rows"], rng)).cuda()
    elif kind == "gradient":
        st["net"] = _network(st["seed"])
        x = torch.from_numpy(_query_rows(case["rows"], rng)).cuda()
        st["theta"] = x[:, :5].contiguous().requires_grad_(True)
        st["rt"], st["choice"] = x[:, 5].contiguous(), x[:, 6].contiguous()
    elif kind == "train":
        st["net"] = net = _network(st["seed"])
        rec, m, v = _training_inputs(case, seed)
        net.m.copy_(torch.from_numpy(m))
        net.v.copy_(torch.from_numpy(v))
        net.step = 1000
        st["records"] = net.prepare_records(torch.from_numpy(rec))
    return st


def run(st):
    kind = st["kind"]
    if kind == "simulate":
        r = st["sim"].simulate(st["theta"], n_samples=st["n"], delta_t=DT, max_t=MAX_T, random_state=st["seed"])
        return {"rts": r["rts"], "choices": r["choices"], "trajectory": r["metadata"]["trajectory"]}
    if kind == "predictive":
        return hssm_support.rng_fn(st["args"], None, np.random.default_rng(st["seed"]), st["fun"], 2)
    if kind == "batch":
        o = st["sim"].run()
        return {"rts": o.rts, "choices": o.choices}
    if kind == "sets":
        o = st["sets"].run(st["seed"])
        return {"rts": o.rts, "choices": o.choices}
    if kind == "records":
        return st["pipe"].run_batch(st["theta"], st["seed"], on_device=True)
    if kind == "kde":
        kb = KdeBatch(st["rts"], st["choices"], st["soff"], [-1, 1])
        ll = kb.evaluate(st["qoff"], st["q"], max_t=MAX_T)
        return {"loglik": ll, "bandwidth": kb.bandwidth, "proportion": kb.proportion}
    if kind == "surrogate":
        return st["net"].forward(st["x"])
    if kind == "gradient":
        ll = st["net"].loglik(st["theta"], st["rt"], st["choice"])
        (g,) = torch.autograd.grad(ll.sum(), st["theta"])
        return {"loglik": ll.detach(), "grad": g}
    if kind == "train":
        net = st["net"]
        loss = net.train_step(st["records"], lr=1e-3)
        return {"loss": loss, "params": net.params, "m": net.m, "v": net.v}
    raise ValueError(kind)


# ---------------------------------------------------------------- work and exact values
def work(case):
    kind = case["kind"]
    if kind in ("simulate", "predictive", "batch", "sets"):
        walks = {"simulate": lambda: case["trials"] * case["samples"], "predictive": lambda: case["trials"],
                 "batch": lambda: case["sets"] * (case["lo"] + case["hi"]) // 2,
                 "sets": lambda: case["sets"] * case["samples"]}[kind]()
        steps = walks * STEPS[case["model"]] * ACCUMULATORS.get(case["model"], 1)
        return {"bytes": 8.0 * walks, "flops": float(STEP_FLOPS * steps)}
    if kind == "records":
        walks = case["sets"] * case["samples"]
        pairs = case["sets"] * 900 * case["samples"] / 2  # 900 evaluated rows against about half of the samples
        return {"bytes": case["sets"] * (1000 * 32.0 + 2 * 384 * 4),
                "flops": STEP_FLOPS * walks * float(STEPS[case["model"]]) + 6.0 * pairs}
    if kind == "kde":
        points, queries = case["sets"] * case["points"], case["sets"] * case["queries"]
        return {"bytes": 8.0 * points + 16.0 * queries, "flops": 6.0 * queries * case["points"] / 2}
    macs = 7 * 100 + 100 * 100 + 100 * 120 + 120
    if kind == "surrogate":
        return {"bytes": 32.0 * case["rows"], "flops": 2.0 * macs * case["rows"]}
    if kind == "gradient":
        return {"bytes": (28.0 + 4.0 + 20.0) * case["rows"], "flops": 4.0 * macs * case["rows"]}
    return {"bytes": 32.0 * case["rows"] + 6 * 4 * 23141.0, "flops": 6.0 * macs * case["rows"]}


def _split(params):
    """The network's layers [(weight, bias), ...] from the flat parameter vector."""
    out, at = [], 0
    for n_in, n_out in ((7, 100), (100, 100), (100, 120), (120, 1)):
        w = params[at:at + n_in * n_out].reshape(n_out, n_in)
        at += n_in * n_out
        out.append((w, params[at:at + n_out]))
        at += n_out
    return out


def _mlp(params, x):
    lo, hi = (torch.tensor(b, dtype=torch.float64, device=x.device) for b in model_config["angle"]["param_bounds"])
    h = torch.cat([(x[:, :5] - (lo + hi) / 2) * (2.0 / (hi - lo)), x[:, 5:]], dim=1)
    layers = _split(params)
    for w, b in layers[:-1]:
        h = torch.tanh(h @ w.T + b)
    w, b = layers[-1]
    return (h @ w.T + b).reshape(-1)


def _initial_params(seed):
    """nn.Linear's default initialisation drawn as the package documents it."""
    rng = np.random.default_rng(seed)
    parts = []
    for n_in, n_out in ((7, 100), (100, 100), (100, 120), (120, 1)):
        k = 1.0 / math.sqrt(n_in)
        parts += [rng.uniform(-k, k, n_in * n_out), rng.uniform(-k, k, n_out)]
    return torch.from_numpy(np.concatenate(parts).astype(np.float32)).double().cuda()


def exact(case, seed):
    kind, rng = case["kind"], np.random.default_rng(seed)
    if kind == "kde":
        return _exact_kde(case, seed)
    if kind == "surrogate":
        x = torch.from_numpy(_query_rows(case["rows"], rng)).cuda().double()
        return torch.cat([_mlp(_initial_params(seed % (2**31 - 1)), c) for c in x.split(65536)])
    if kind == "gradient":
        x = torch.from_numpy(_query_rows(case["rows"], rng)).cuda().double()
        params, ll, grad = _initial_params(seed % (2**31 - 1)), [], []
        for c in x.split(65536):
            th = c[:, :5].clone().requires_grad_(True)
            out = _mlp(params, torch.cat([th, c[:, 5:]], dim=1))
            grad.append(torch.autograd.grad(out.sum(), th)[0])
            ll.append(out.detach())
        return {"loglik": torch.cat(ll), "grad": torch.cat(grad)}
    if kind == "train":
        rec, m, v = (torch.from_numpy(a).double().cuda() for a in _training_inputs(case, seed))
        params = _initial_params(seed % (2**31 - 1)).requires_grad_(True)
        label = rec[:, 7].clamp(min=math.log(1e-7))
        loss = torch.nn.functional.huber_loss(_mlp(params, rec[:, :7]), label)
        (g,) = torch.autograd.grad(loss, params)
        m, v, step = 0.9 * m + 0.1 * g, 0.999 * v + 0.001 * g * g, 1001
        upd = 1e-3 * (m / (1 - 0.9**step)) / (torch.sqrt(v / (1 - 0.999**step)) + 1e-8)
        return {"loss": loss.detach(), "params": (params - upd).detach(), "m": m, "v": v}
    return None  # simulated trajectories and what is resampled from them are random draws


def _exact_kde(case, seed):
    rts, choices, soff, qoff, q = _kde_inputs(case, seed)
    if case["sets"] * case["queries"] * case["points"] > 4e9:
        return None
    ll = torch.empty_like(q)
    bw, prop = [], []
    for s in range(case["sets"]):
        r, c = rts[soff[s]:soff[s + 1]].double(), choices[soff[s]:soff[s + 1]]
        for j, value in enumerate((-1, 1)):
            grp = 2 * s + j
            mine = c == value
            x = torch.log(r[mine & (r != -999.0)])
            n, p = x.numel(), float(mine.double().mean())
            h = (4.0 / (3.0 * n)) ** 0.2 * max(float(x.std(unbiased=False)), 1e-3)
            lq = torch.log(q[qoff[grp]:qoff[grp + 1]].clamp(min=1e-4))
            for at in range(0, lq.numel(), 512):
                part = lq[at:at + 512]
                e = -((part[:, None] - x[None, :]) ** 2) / (2 * h * h)
                v = (math.log(p) - math.log(n) - math.log(h) - 0.5 * math.log(2 * math.pi)
                     + torch.logsumexp(e, dim=1) - part)
                lo = int(qoff[grp]) + at
                ll[lo:lo + part.numel()] = torch.where(v > -66.774, v, torch.full_like(v, -66.774))
            bw.append(h)
            prop.append(p)
    return {"loglik": ll, "bandwidth": np.asarray(bw), "proportion": np.asarray(prop)}
