"""The work users of this engine have it do, as cases that can be timed.

Every case goes through the public entry points (hawkes_b200: CudaHawkes,
Multiset, Sampler) from host arrays to host results, the way the reference's
callers use its engine: the R API and its timing function, the MCMC sampler,
the BEAST binding, the command-line benchmark.  Event sets come from
hawkes_b200.workloads (uniform box, uneven sets, clustered process) and from
the reference's timing function (standard normal locations, times 1..N);
parameters are log-normal around the sampler's defaults, as in the proposals
workload.

A case is one of these kinds:

  evaluate  new parameters (all six), log-likelihood and gradient, on events the
            engine holds: one optimiser, HMC or Metropolis step that moves tauX
            or tauT.  probs also reads the per-event probabilities.
  data      the same from new host events each time: setTimesData,
            updateLocations, setParameters, log-likelihood and gradient.
  timetest  the reference's timeTest(): N(0, 1) locations, times 1..N,
            Exp(1) parameters, the log-likelihood only.
  proposals K parameter vectors on one event set in one call.
  sets      several event sets of uneven size, new data for each, one call.
  mcmc      the reference sampler's steps at fixed tauX and tauT (sigma, omega,
            theta and mu0 proposed in turn), then one location proposal that is
            rejected: the BEAST binding's store, move, evaluate, restore.
  chains    a short run of the sampler's device driver, several chains.

Results are handed on in the precision of the engine mode: double precision in
the FP64 mode; in the two single-precision modes the log-likelihood stays a
double where it is compensated (an acceptance test subtracts two of them), and
gradients and probabilities go into single-precision arrays, as the parameters
of a single-precision optimiser take them.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import hawkes_b200 as hb
from hawkes_b200 import workloads

_MODES = {
    "fp64": hb.CUDA,
    "fp32c": hb.CUDA | hb.COMPENSATED,
    "float": hb.CUDA | hb.FLOAT,
}


def listed():
    return [
        # The smallest evaluations: a few hundred events, where a call is launches
        # and latency (the JNI singleton, examples, short series).
        {"name": "evaluate_fp64_n500", "kind": "evaluate", "mode": "fp64", "N": 500, "D": 2,
         "events": "uniform", "probs": True},
        # The reference's own timing function at its default size.
        {"name": "timetest_fp64_n5000", "kind": "timetest", "mode": "fp64", "N": 5000, "D": 2},
        # Three space dimensions, an odd size, probabilities read back.
        {"name": "evaluate_fp32c_d3_n12001", "kind": "evaluate", "mode": "fp32c", "N": 12001,
         "D": 3, "events": "uniform", "probs": True},
        # The reference's single precision on a mid-sized set.
        {"name": "evaluate_float_n50000", "kind": "evaluate", "mode": "float", "N": 50000, "D": 2,
         "events": "uniform", "probs": False},
        # The headline workload in double precision and FP32-compensated.
        {"name": "evaluate_fp64_n100000", "kind": "evaluate", "mode": "fp64", "N": 100000, "D": 2,
         "events": "uniform", "probs": False},
        {"name": "evaluate_fp32c_n100000", "kind": "evaluate", "mode": "fp32c", "N": 100000,
         "D": 2, "events": "uniform", "probs": False},
        # The same end to end from new host events.
        {"name": "data_fp32c_n100000", "kind": "data", "mode": "fp32c", "N": 100000, "D": 2,
         "events": "uniform"},
        # Batched proposals of parallel chains that move every parameter.
        {"name": "proposals_fp32c_n20000_k64", "kind": "proposals", "mode": "fp32c", "N": 20000,
         "D": 2, "K": 64},
        # Many regions or simulated data sets of uneven size, new data for each.
        {"name": "sets_fp32c_s24", "kind": "sets", "mode": "fp32c", "S": 24, "D": 2, "lo": 1000,
         "hi": 50000},
        # The largest: a clustered branching process over a wide box.
        {"name": "evaluate_fp32c_clustered_n500000", "kind": "evaluate", "mode": "fp32c",
         "N": 500000, "D": 2, "events": "clustered", "probs": False},
        # One round of the sampler's steps and a location proposal on the headline
        # events.
        {"name": "mcmc_fp32c_n100000", "kind": "mcmc", "mode": "fp32c", "N": 100000, "D": 2},
        # A short device-driven sampler run on a few thousand events.
        {"name": "chains_fp64_n3000_c16", "kind": "chains", "mode": "fp64", "N": 3000, "D": 2,
         "chains": 16, "iterations": 40},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["evaluate", "evaluate", "evaluate", "data", "timetest", "proposals", "sets",
                       "mcmc", "chains"])
    mode = rng.choice(["fp64", "fp32c", "fp32c", "fp64", "float"])
    if kind == "evaluate":
        D = rng.choice([1, 2, 2, 2, 2, 3, 4, 8])
        events = rng.choice(["uniform", "uniform", "clustered"]) if D == 2 else "uniform"
        top = {"fp64": 150000, "fp32c": 300000, "float": 300000}[mode] if D <= 2 else 60000
        return {"kind": kind, "mode": mode, "N": _log_int(rng, 300, top), "D": D,
                "events": events, "probs": rng.random() < 0.5}
    if kind == "data":
        D = rng.choice([2, 2, 3])
        return {"kind": kind, "mode": mode, "N": _log_int(rng, 1000, 120000 if D == 2 else 40000),
                "D": D, "events": "uniform"}
    if kind == "timetest":
        return {"kind": kind, "mode": rng.choice(["fp64", "float"]),
                "N": _log_int(rng, 500, 100000), "D": 2}
    if kind == "proposals":
        mode = rng.choice(["fp64", "fp32c"])
        N = _log_int(rng, 1000, 20000)
        return {"kind": kind, "mode": mode, "N": N, "D": 2, "K": rng.randint(8, 64)}
    if kind == "sets":
        lo = _log_int(rng, 200, 3000)
        return {"kind": kind, "mode": rng.choice(["fp64", "fp32c"]), "S": rng.randint(6, 32),
                "D": 2, "lo": lo, "hi": lo * rng.randint(4, 20)}
    if kind == "mcmc":
        return {"kind": kind, "mode": rng.choice(["fp64", "fp32c"]),
                "N": _log_int(rng, 2000, 120000), "D": 2}
    return {"kind": kind, "mode": rng.choice(["fp64", "fp32c"]), "N": _log_int(rng, 500, 8000),
            "D": 2, "chains": rng.randint(4, 16), "iterations": rng.randint(20, 60)}


# ------------------------------------------------------------------ inputs --

def _events(case, seed):
    if case["events"] == "clustered":
        n = case["N"]
        # the density of the 500,000-event configuration: the box grows with N
        return workloads.clustered(N=n, seed=seed, background=n // 2 + 50,
                                   oversample=0.04 if n > 20000 else 0.5,
                                   box=50.0 * math.sqrt(n / 500000.0) + 2.0)
    return workloads.uniform(case["N"], seed, D=case["D"])


def _inputs(case, seed):
    """Everything prepare() and exact() need, from the seed alone."""
    kind = case["kind"]
    rng = np.random.default_rng([seed, 77])
    base = np.asarray(workloads.BASE_PARAMS)
    if kind == "sets":
        sets = workloads.uneven(case["S"], seed, lo=case["lo"], hi=case["hi"], D=case["D"])
        return {"sets": sets, "params": np.stack([p for _, _, p in sets])}
    if kind == "timetest":
        n = case["N"]
        loc = rng.standard_normal((n, case["D"]))
        t = np.arange(1, n + 1, dtype=np.float64)
        return {"loc": loc, "t": t, "params": rng.exponential(1.0, size=6) + 0.05}
    if kind in ("evaluate", "data"):
        loc, t = _events(case, seed)
    else:
        loc, t = workloads.uniform(case["N"], seed, D=case["D"])
    if kind in ("evaluate", "data"):
        return {"loc": loc, "t": t, "start": base, "params": workloads.proposals(1, seed)[0]}
    if kind == "proposals":
        return {"loc": loc, "t": t, "params": workloads.proposals(case["K"], seed)}
    if kind == "mcmc":
        steps, p = [], base.copy()
        for k, f in zip((0, 3, 4, 5), np.exp(0.1 * rng.standard_normal(4))):
            p = p.copy()
            p[k] *= f
            steps.append(p)
        k = int(rng.integers(0, case["N"]))
        return {"loc": loc, "t": t, "start": base, "steps": steps, "moved": k,
                "to": loc[k] + rng.normal(0.0, 0.5, size=case["D"])}
    z = rng.standard_normal((case["chains"], 6))
    z[:, 1:3] = 0.0  # the sampler keeps tauX and tauT fixed
    return {"loc": loc, "t": t, "start": base, "init": base * np.exp(0.1 * z), "seed": seed}


def prepare(case, seed):
    """An engine that holds the events and has been evaluated once, as in a
    running program; the inputs of the next step beside it."""
    x = dict(_inputs(case, seed), kind=case["kind"], mode=case["mode"], probs=case.get("probs"),
             iterations=case.get("iterations"))
    flags = _MODES[case["mode"]]
    if case["kind"] == "sets":
        eng = hb.Multiset(case["D"], [len(t) for _, t, _ in x["sets"]], flags, 0)
        for s, (loc, t, _) in enumerate(x["sets"]):
            eng.setData(s, loc, t)
        eng.logLikelihoodAndGradient(x["params"])
        x["engine"] = eng
        return x
    if case["kind"] == "timetest":
        flags |= hb.NO_INCREMENTAL  # every evaluation in full, as timeTest() does
    eng = hb.CudaHawkes(case["D"], len(x["t"]), flags, 0)
    eng.setTimesData(x["t"])
    eng.updateLocations(-1, x["loc"])
    start = x.get("start", x["params"] if case["kind"] == "timetest" else workloads.BASE_PARAMS)
    eng.setParameters(start)
    if case["kind"] == "proposals":
        eng.batchLogLikelihoodAndGradient(x["params"])
    else:
        eng.getLogLikelihoodAndGradient()
    x["engine"] = eng
    return x


# --------------------------------------------------------------- one pass --

def _handed_on(mode, loglik, *arrays):
    """(loglik, arrays) in the mode's precision (see the module's text)."""
    if mode == "fp64":
        return (loglik, *arrays)
    if mode == "float":
        loglik = np.float32(loglik)
    return (loglik, *[np.asarray(a, dtype=np.float32) for a in arrays])


def run(x):
    eng, kind, mode = x["engine"], x["kind"], x["mode"]
    if kind == "evaluate":
        # the step from the current point and back: each of the two moves tauX and
        # tauT, so each is a full evaluation
        eng.setParameters(x["start"])
        ll0, g0 = eng.getLogLikelihoodAndGradient()
        eng.setParameters(x["params"])
        ll, g = eng.getLogLikelihoodAndGradient()
        out = _handed_on(mode, ll0, g0) + _handed_on(mode, ll, g)
        return out + _handed_on(mode, 0.0, eng.getProbsSelfExcite())[1:] if x["probs"] else out
    if kind == "data":
        eng.setTimesData(x["t"])
        eng.updateLocations(-1, x["loc"])
        eng.setParameters(x["params"])
        return _handed_on(mode, *eng.getLogLikelihoodAndGradient())
    if kind == "timetest":
        eng.setParameters(x["params"])
        return _handed_on(mode, eng.getSumOfLikContribs())[0]
    if kind == "proposals":
        return _handed_on(mode, *eng.batchLogLikelihoodAndGradient(x["params"]))
    if kind == "sets":
        for s, (loc, t, _) in enumerate(x["sets"]):
            eng.setData(s, loc, t)
        return _handed_on(mode, *eng.logLikelihoodAndGradient(x["params"]))
    if kind == "mcmc":
        lls = []
        for p in x["steps"]:
            eng.setParameters(p)
            lls.append(eng.getSumOfLikContribs())
        eng.storeState()
        eng.updateLocations(x["moved"], x["to"])
        lls.append(eng.getSumOfLikContribs())
        eng.restoreState()
        return np.array(lls)
    with hb.Sampler(x["init"], radius=0.3, seed=x["seed"]) as s:
        samples, targets = s.run(eng, x["iterations"], device=True)
    return samples, targets


# ------------------------------------------------------------------- work --

def work(case):
    """Bytes: events and parameters in, results out.  Floating-point operations:
    of the direct sum over unordered pairs, 3 D + 30 for a pair's terms and their
    weighted sums (an exponential counted as 10)."""
    D, per = case["D"], 3 * case["D"] + 30
    kind = case["kind"]

    def pairs(n):
        return 0.5 * n * (n + 1.0)

    if kind == "sets":
        # sizes are log-uniform in [lo, hi]
        lo, hi, S = case["lo"], case["hi"], case["S"]
        mean = (hi - lo) / math.log(hi / lo)
        mean2 = (hi * hi - lo * lo) / (2.0 * math.log(hi / lo))
        return {"bytes": 8.0 * S * (mean * (D + 1) + 13), "flops": per * S * 0.5 * (mean2 + mean)}
    n = case["N"]
    events = 8.0 * n * (D + 1)
    if kind == "proposals":
        return {"bytes": events + 8.0 * 13 * case["K"], "flops": per * case["K"] * pairs(n)}
    if kind == "mcmc":
        # two steps of the self-excitation sums, then O(N) updates
        return {"bytes": events + 8.0 * (6 * n + 13 * 5), "flops": 2.0 * (per / 2) * pairs(n)}
    if kind == "chains":
        return {"bytes": events + 8.0 * 7 * case["chains"] * case["iterations"],
                "flops": (per / 2) * pairs(n) * case["chains"] * case["iterations"]}
    outputs = 13 + (n if case.get("probs") else 0)
    return {"bytes": events + 8.0 * outputs,
            "flops": (2.0 if kind == "evaluate" else 1.0) * per * pairs(n)}


# ------------------------------------------------------------------ exact --

def _exact_eval(loc, t, p):
    """(log-likelihood, gradient, probabilities) in 64 bits, by the model's
    formulas (src/NewHawkes.hpp:520-547, :636-660) over all ordered pairs."""
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    x = torch.as_tensor(np.asarray(loc, dtype=np.float64), device=dev)
    s = torch.as_tensor(np.asarray(t, dtype=np.float64), device=dev)
    N, D = x.shape
    sigma, a, b, omega, theta, mu0 = (float(v) for v in p)
    rows = max(1, min(N, 80_000_000 // N))
    sums = torch.empty((6, N), dtype=torch.float64, device=dev)
    for i in range(0, N, rows):
        xi, ti = x[i:i + rows], s[i:i + rows]
        dt = ti[:, None] - s[None, :]
        d2 = torch.zeros_like(dt)
        for k in range(D):
            d2 += (xi[:, k, None] - x[None, :, k]).square_()
        t2 = dt.square()
        B = torch.exp((d2 * (-0.5 * a * a)).add_(t2, alpha=-0.5 * b * b))
        sums[0, i:i + rows] = B.sum(1)
        sums[1, i:i + rows] = torch.linalg.vecdot(B, d2)
        sums[2, i:i + rows] = torch.linalg.vecdot(B, t2)
        del B, t2
        S = torch.exp((d2 * (-0.5 * sigma * sigma)).add_(dt, alpha=-omega)
                      .masked_fill_(dt <= 0, -math.inf))
        sums[3, i:i + rows] = S.sum(1)
        sums[4, i:i + rows] = torch.linalg.vecdot(S, d2)
        sums[5, i:i + rows] = torch.linalg.vecdot(S, dt)
        del S, d2, dt
    Sb, Sbd, Sbt, Ss, Ssd, Sst = sums
    fB = a ** D * b / (2 * math.pi)
    fS = omega * sigma ** D / math.sqrt(2 * math.pi)
    lam = mu0 * fB * Sb + theta * fS * Ss
    rest = s[-1] - s

    def cdf(v):
        return 0.5 * torch.erfc(-v / math.sqrt(2.0))

    def pdf(v):
        return torch.exp(-0.5 * v * v) / math.sqrt(2 * math.pi)

    decay = torch.exp(-omega * rest)
    mass = cdf(b * rest) - cdf(-b * s)
    ll = torch.log(lam) + theta * (decay - 1) - mu0 * mass
    g = torch.stack([
        (theta * fS * (D / sigma * Ss - sigma * Ssd) / lam).sum(),
        (mu0 * fB * (D / a * Sb - a * Sbd) / lam).sum(),
        (mu0 * fB * (Sb / b - b * Sbt) / lam
         - mu0 * (pdf(b * rest) * rest + pdf(b * s) * s)).sum(),
        (theta * fS * (Ss / omega - Sst) / lam - theta * rest * decay).sum(),
        (fS * Ss / lam + decay - 1).sum(),
        (fB * Sb / lam - mass).sum(),
    ])
    total = float(ll.sum()) + N * (D - 1) * math.log(1 / math.sqrt(2 * math.pi))
    return total, g.cpu().numpy(), (theta * fS * Ss / lam).cpu().numpy()


def exact(case, seed):
    kind = case["kind"]
    if kind == "chains":
        return None  # a chain's path is decided by its acceptance tests, not by one formula
    pairs = {"proposals": lambda: case["K"] * float(case["N"]) ** 2,
             "sets": lambda: case["S"] * float(case["hi"]) ** 2 / 4.0}
    if pairs.get(kind, lambda: float(case["N"]) ** 2)() > 1.5e11:
        return None  # takes too long
    x = _inputs(case, seed)
    if kind == "evaluate":
        ll0, g0, _ = _exact_eval(x["loc"], x["t"], x["start"])
        ll, g, probs = _exact_eval(x["loc"], x["t"], x["params"])
        return (ll0, g0, ll, g, probs) if case["probs"] else (ll0, g0, ll, g)
    if kind == "data":
        return _exact_eval(x["loc"], x["t"], x["params"])[:2]
    if kind == "timetest":
        return _exact_eval(x["loc"], x["t"], x["params"])[0]
    if kind == "proposals":
        r = [_exact_eval(x["loc"], x["t"], p) for p in x["params"]]
        return np.array([v[0] for v in r]), np.stack([v[1] for v in r])
    if kind == "sets":
        r = [_exact_eval(loc, t, p) for loc, t, p in x["sets"]]
        return np.array([v[0] for v in r]), np.stack([v[1] for v in r])
    lls = [_exact_eval(x["loc"], x["t"], p)[0] for p in x["steps"]]
    moved = x["loc"].copy()
    moved[x["moved"]] = x["to"]
    return np.array(lls + [_exact_eval(moved, x["t"], x["steps"][-1])[0]])
