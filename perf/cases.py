"""The work a user of this package has it do, as measurable cases through its public entry points.

Every case is one call (or the few calls that belong together) on data of the distributions the
path meets in earnest: complete nested-sampling runs from a model and a key to the results,
batches of independent runs, linear-regression evidence problems, the reweighted-evidence
adjoint, the evidence of a stored sample set, simulated evidences, and the model's forward and
prior-transform passes over many points.
"""
import ctypes
import math

import numpy as np
import torch

import jaxns_gb300 as gb
from jaxns_gb300 import binding, engine
from jaxns_gb300.adjoint import DeadSet, EvidenceFn
from jaxns_gb300.batched import BatchedNestedSampler
from jaxns_gb300.engine import NSBatch

DEVICE = "cuda"


# ------------------------------------------------------------------------- the cases

def listed():
    return [
        # one run of the reference's published benchmark (D = 8, 0.99 correlations, a shifted
        # MultivariateNormalTriL prior) at the defaults, from key to results: what a new user types
        dict(name="call_gh168", kind="call", family="tril", D=8, live=0, slices=0, phantoms=False, guided=False),
        # one run for parameter estimation on a correlated Gaussian: phantom samples, the
        # warp-cooperative sampler, one problem on the whole device
        dict(name="call_mvn_d24_phantoms", kind="call", family="mvn", D=24, live=0, slices=0, phantoms=True,
             guided=False),
        # the headline batch: 1024 seeds of the Gaussian shells, D = 10, 1000 live points, 50 slices
        dict(name="batch_shells_d10", kind="batch", family="shells", D_lo=10, D_hi=10, runs=1024, live=1000, slices=50,
             iterations=0),
        # a few dozen seeds of the published benchmark: a repeatability study
        dict(name="batch_gh168_48", kind="batch", family="tril", D_lo=8, D_hi=8, runs=48, live=240, slices=40,
             iterations=0),
        # many models of uneven dimension in one batch (50 D live points, 5 D slices), its first
        # iterations
        dict(name="batch_mvn_mixed", kind="batch", family="mvn", D_lo=2, D_hi=64, runs=64, live=0, slices=0,
             iterations=3),
        # Bayesian linear regression with 4096 rows and 32 columns, 1024 live points: the first 48
        # iterations of one problem
        dict(name="blr_4096x32", kind="blr", N=4096, P=32, runs=1, live=1024, iterations=48),
        # twelve linear-regression problems of uneven size in one batch (up to 16384 x 64)
        dict(name="blr_batch_12", kind="blr", N=16384, P=64, runs=12, live=0, iterations=2),
        # evidence and gradient of the linear regression over one run's dead points, as an
        # optimiser of its hyperparameters calls it: autograd forward and backward
        dict(name="adjoint_40k_4096x32", kind="adjoint", M=40000, N=4096, P=32),
        # live-point counts and evidence of one long run's stored samples
        dict(name="evidence_250k", kind="evidence", N=250000, live=2000, phantoms=False),
        # the default 100 simulated evidences of a run with 22000 samples
        dict(name="sample_evidence_22k", kind="sample", M=22000, S=100),
        # the model's log likelihood over a large set of points
        dict(name="forward_mvn_d64", kind="forward", family="mvn", D=64, B=200000, N=0),
        # samples and posterior densities of a merged set of runs with a MultivariateNormalTriL prior
        dict(name="transform_tril_d8", kind="transform", D=8, rows=500000, tril=True, double=False),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["call", "call", "batch", "batch", "mixed", "blr", "blr", "adjoint", "evidence", "sample",
                       "forward", "transform"])
    if kind == "call":
        family = rng.choice(["tril", "mvn", "shells"])
        D = _log_int(rng, 2, 24)
        return dict(kind="call", family=family, D=D, live=rng.choice([0, rng.randint(60, 900)]),
                    slices=rng.choice([0, rng.randint(2 * D, 5 * D)]), phantoms=rng.random() < 0.3,
                    guided=rng.random() < 0.15)
    if kind == "batch":
        D = rng.randint(2, 16)
        return dict(kind="batch", family=rng.choice(["tril", "mvn", "shells"]), D_lo=D, D_hi=D,
                    runs=_log_int(rng, 4, 400), live=rng.randint(100, 1000), slices=rng.randint(2 * D, 5 * D),
                    iterations=0)
    if kind == "mixed":
        return dict(kind="batch", family="mvn", D_lo=rng.randint(2, 20), D_hi=rng.randint(24, 64),
                    runs=_log_int(rng, 8, 60), live=0, slices=0, iterations=rng.randint(1, 3))
    if kind == "blr":
        P = rng.randint(4, 64)
        return dict(kind="blr", N=_log_int(rng, 300, 16384), P=P, runs=_log_int(rng, 1, 10),
                    live=rng.choice([0, rng.randint(100, 1200)]), iterations=rng.randint(1, 4))
    if kind == "adjoint":
        return dict(kind="adjoint", M=_log_int(rng, 1000, 80000), N=_log_int(rng, 256, 10000), P=rng.randint(4, 64))
    if kind == "evidence":
        return dict(kind="evidence", N=_log_int(rng, 2000, 600000), live=_log_int(rng, 100, 4000),
                    phantoms=rng.random() < 0.3)
    if kind == "sample":
        return dict(kind="sample", M=_log_int(rng, 1000, 100000), S=_log_int(rng, 10, 300))
    if kind == "forward":
        family = rng.choice(["mvn", "shells", "lingauss"])
        lg = family == "lingauss"
        return dict(kind="forward", family=family, D=rng.randint(2, 64), B=_log_int(rng, 500, 20000 if lg else 500000),
                    N=_log_int(rng, 256, 4096) if lg else 0)
    return dict(kind="transform", D=rng.randint(1, 40), rows=_log_int(rng, 1000, 500000), tril=rng.random() < 0.4,
                double=rng.random() < 0.3)


# ------------------------------------------------------------------------- models

def _generator(seed, *more):
    return np.random.default_rng([int(seed) & 0x7fffffff, *more])


def _cov(g, D):
    A = g.standard_normal((D, D))
    return A @ A.T / D + 0.1 * np.eye(D)


def _model(family, D, g):
    """The three sampled models: a correlated Gaussian under a Uniform(-10, 10) prior, the published
    benchmark's Gaussian under a MultivariateNormalTriL(15, I) prior, and two Gaussian shells."""
    if family == "mvn":
        prior = gb.Uniform(-10.0 * np.ones(D), 10.0 * np.ones(D))
        like = gb.MultivariateNormalLikelihood(g.standard_normal(D), _cov(g, D))
    elif family == "tril":
        prior = gb.MultivariateNormalTriL(15.0 * np.ones(D), np.eye(D))
        like = gb.MultivariateNormalLikelihood(np.zeros(D), np.where(np.eye(D) == 1, 1.0, 0.99))
    else:
        prior = gb.Uniform(-6.0 * np.ones(D), 6.0 * np.ones(D))
        c = np.zeros(D)
        c[0] = 3.5
        like = gb.GaussianShellsLikelihood(c, -c, 2.0, 0.1)

    def prior_model():
        x = yield gb.Prior(prior, name="x")
        return x

    return gb.Model(prior_model, like)


def _blr_problem(g, N, P, sigma, tau):
    Phi = g.standard_normal((N, P), dtype=np.float32)
    y = (Phi.astype(np.float64) @ g.standard_normal(P) + sigma * g.standard_normal(N)).astype(np.float32)

    def prior_model():
        w = yield gb.Prior(gb.Normal(np.zeros(P), tau * np.ones(P)), name="w")
        return w

    return gb.Model(prior_model, gb.LinearGaussianLikelihood(Phi, y, sigma)), Phi, y


def _mixed_dims(case):
    g = np.random.default_rng([case["D_lo"], case["D_hi"], case["runs"]])
    return [int(d) for d in g.integers(case["D_lo"], case["D_hi"] + 1, size=case["runs"])]


def _blr_dims(case):
    """The sizes of a batch's problems: the first is the case's own, the others spread below it."""
    g = np.random.default_rng([case["N"], case["P"], case["runs"]])
    R = case["runs"] - 1
    Ns = g.integers(max(64, case["N"] // 16), case["N"] + 1, size=R)
    Ps = g.integers(max(2, case["P"] // 6), case["P"] + 1, size=R)
    return [(case["N"], case["P"])] + [(int(n), int(p)) for n, p in zip(Ns, Ps)]


def _keys(seed, R):
    return np.array([gb.random.PRNGKey((int(seed) & 0x7fffffff) * 4096 + r) for r in range(R)], np.uint32)


# ------------------------------------------------------------------------- prepare

def prepare(case, seed):
    return {"kind": case["kind"], **globals()["_prepare_" + case["kind"]](case, seed)}


def _prepare_call(case, seed):
    model = _model(case["family"], case["D"], _generator(seed, 1))
    ns = gb.NestedSampler(model, num_live_points=case["live"] or None, num_slices=case["slices"] or None,
                          parameter_estimation=case["phantoms"], gradient_guided=case["guided"])
    rows, D = ns.nested_sampler.max_samples, case["D"]
    table = lambda *shape, dtype=torch.float64: torch.zeros(rows, *shape, dtype=dtype, device=DEVICE)
    tables = {"x": table(D), "U_samples": table(D, dtype=torch.float32), "log_L_samples": table(),
              "log_dp_mean": table(), "log_X_mean": table(), "log_posterior_density": table(),
              "num_live_points_per_sample": table(dtype=torch.int64),
              "num_likelihood_evaluations_per_sample": table(dtype=torch.int64)}
    return {"ns": ns, "key": gb.random.PRNGKey(seed), "tables": tables}


def _prepare_batch(case, seed):
    samplers, model = [], None
    for r, D in enumerate(_mixed_dims(case)):
        if model is None or case["D_lo"] != case["D_hi"]:  # one model and many keys, or many models
            model = _model(case["family"], D, _generator(seed, 2, r))
        samplers.append(gb.NestedSampler(model, num_live_points=case["live"] or 50 * D,
                                         num_slices=case["slices"] or 5 * D))
    tc = gb.TerminationCondition(dlogZ=1e-4)
    return {"bns": BatchedNestedSampler(samplers, _keys(seed, len(samplers)), [tc] * len(samplers)),
            "iterations": case["iterations"]}


def _prepare_blr(case, seed):
    samplers = []
    for r, (N, P) in enumerate(_blr_dims(case)):
        model, _, _ = _blr_problem(_generator(seed, 3, r), N, P, 0.5, 1.0)
        live = case["live"] or 25 * P
        H = 0.5 * P * math.log(1.0 + N / 0.25)
        samplers.append(gb.NestedSampler(model, num_live_points=live, max_samples=int(live * (1.3 * H + 2 * P + 60))))
    return {"bns": BatchedNestedSampler(samplers, _keys(seed, len(samplers)), store_U=True),
            "iterations": case["iterations"]}


def _dead_points(case, seed):
    """Dead points of a run on y ~ N(Phi w, 0.25 I), w ~ N(0, I): balls around the posterior mean that
    shrink by the run's compression, and the log prior mass of each."""
    g = _generator(seed, 4)
    M, N, P = case["M"], case["N"], case["P"]
    _, Phi, y = _blr_problem(g, N, P, 0.5, 1.0)
    G = Phi.astype(np.float64).T @ Phi.astype(np.float64) / 0.25 + np.eye(P)
    mean = np.linalg.solve(G, Phi.astype(np.float64).T @ y.astype(np.float64) / 0.25)
    width = 1.0 / math.sqrt(N / 0.25)
    tg = torch.Generator(device=DEVICE).manual_seed(int(seed) & 0x7fffffff)
    f = torch.arange(M, device=DEVICE, dtype=torch.float64) / M
    radius = torch.exp(math.log(0.5 * width) * f)
    w = torch.as_tensor(mean, device=DEVICE) + radius[:, None] * torch.randn(M, P, generator=tg, device=DEVICE,
                                                                          dtype=torch.float64)
    U = torch.special.ndtr(w).clamp(1e-14, 1.0 - 1e-14)
    n = M / (P * math.log(2.0 / width))
    log_w = -torch.arange(M, device=DEVICE, dtype=torch.float64) / n - math.log(n)
    dev = lambda x: torch.as_tensor(x, device=DEVICE)
    return DeadSet(U=U.contiguous(), log_w=log_w, Phi=dev(Phi).contiguous(), y=dev(y).contiguous())


def _prepare_adjoint(case, seed):
    theta = torch.tensor([0.05 + 0.001 * (seed % 7), math.log(0.52)], dtype=torch.float64, device=DEVICE)
    return {"ds": _dead_points(case, seed), "theta": theta}


def _sample_set(case, seed):
    """A static run's stored samples: shells of n / 2 discards replaced by draws above the contour,
    log L of a Gaussian peak; with phantoms, a third of the store sits one shell late (out of order)."""
    g = _generator(seed, 5)
    N, n = case["N"], min(case["live"], max(2, case["N"] // 2))
    s = max(1, n // 2)
    live, sender = np.sort(-g.standard_exponential(n))[::-1].copy(), np.zeros(n, np.int64)  # log X, descending
    out_x, out_s, total = [], [], 0
    while total + s + n <= N:
        out_x.append(live[:s])
        out_s.append(sender[:s])
        total += s
        new = live[s - 1] - g.standard_exponential(s)
        x = np.concatenate([new, live[s:]])
        sd = np.concatenate([np.full(s, total - 1), sender[s:]])
        order = np.argsort(-x, kind="stable")
        live, sender = x[order], sd[order]
    k = min(n, N - total)
    log_X = np.concatenate(out_x + [live[:k]])
    senders = np.concatenate(out_s + [sender[:k]])
    dim = max(2.0, N / n / 4.0)
    log_L = (-50.0 * dim * np.exp(2.0 * log_X / dim)).astype(np.float32)
    if case["phantoms"]:
        m = len(log_L) // 3
        at = np.sort(g.choice(len(log_L), size=m, replace=False))
        order = np.argsort(np.arange(len(log_L)) + np.where(np.isin(np.arange(len(log_L)), at), s, 0), kind="stable")
        log_L, senders = log_L[order], senders[order]
    return log_L, senders.astype(np.int32), n


def _prepare_evidence(case, seed):
    log_L, sender, n = _sample_set(case, seed)
    dev = lambda x: torch.as_tensor(x, device=DEVICE)
    return {"lib": binding.bind(), "log_L": dev(log_L), "sender": dev(sender), "nmax": n + 64,
            "ncoef": dev(engine.ncoef_table(n + 64))}


def _simulated_run(case, seed):
    log_L, _, n = _sample_set(dict(N=case["M"], live=max(50, case["M"] // 20), phantoms=False), seed)
    counts = np.concatenate([np.full(len(log_L) - n, n), np.arange(n, 0, -1)]).astype(np.int32)
    return counts, np.sort(log_L).astype(np.float64)


def _prepare_sample(case, seed):
    counts, log_L = _simulated_run(case, seed)
    return {"key": gb.random.PRNGKey(seed), "counts": torch.as_tensor(counts, device=DEVICE),
            "log_L": torch.as_tensor(log_L, device=DEVICE), "S": case["S"]}


def _points(seed, B, D, dtype):
    tg = torch.Generator(device=DEVICE).manual_seed(int(seed) & 0x7fffffff)
    return torch.rand(B, D, generator=tg, device=DEVICE, dtype=torch.float64).clamp(1e-9, 1.0 - 1e-7).to(dtype)


def _prepare_forward(case, seed):
    g = _generator(seed, 6)
    lg = case["family"] == "lingauss"
    model = _blr_problem(g, case["N"], case["D"], 0.5, 1.0)[0] if lg else _model(case["family"], case["D"], g)
    ns = gb.NestedSampler(model, num_live_points=64, num_slices=2)
    batch = NSBatch([ns.nested_sampler.run_spec(gb.random.PRNGKey(seed), ns.normalise_term_cond(None))])
    return {"batch": batch, "U": _points(seed, case["B"], case["D"], torch.float64 if lg else torch.float32)}


def _transform_model(case, seed):
    g = _generator(seed, 7)
    D = case["D"]
    half = D // 2

    def prior_model():
        if case["tril"]:
            yield gb.Prior(gb.MultivariateNormalTriL(g.standard_normal(D), np.linalg.cholesky(_cov(g, D))), name="x")
        else:
            if half:
                yield gb.Prior(gb.Uniform(-3.0 * np.ones(half), 5.0 * np.ones(half)), name="a")
            yield gb.Prior(gb.Normal(np.ones(D - half), 2.0 * np.ones(D - half)), name="b")

    return gb.Model(prior_model, gb.MultivariateNormalLikelihood(np.zeros(D), np.eye(D)))


def _prepare_transform(case, seed):
    U = _points(seed, case["rows"], case["D"], torch.float64 if case["double"] else torch.float32)
    log_L = -torch.rand(case["rows"], device=DEVICE, dtype=torch.float64,
                        generator=torch.Generator(device=DEVICE).manual_seed(int(seed) & 0x7fffffff)) * 40.0
    return {"model": _transform_model(case, seed), "U": U, "log_L": log_L}


# ------------------------------------------------------------------------- run

def run(state):
    return globals()["_run_" + state["kind"]](state)


def _run_call(st):
    reason, state = st["ns"](st["key"], gb.TerminationCondition(dlogZ=1e-4))
    res = st["ns"].to_results(reason, state)._asdict()
    for name, table in st["tables"].items():  # the user's own tables: runs differ in their sample counts
        table[:res["total_num_samples"]] = res["samples"]["x"] if name == "x" else res[name]
    scalars = {k: v for k, v in res.items() if isinstance(v, (int, float))}
    return {**scalars, **st["tables"]}


def _run_batch(st):
    bns = st["bns"]
    if st["iterations"]:
        reasons = bns(max_iterations=st["iterations"], check=False)
    else:
        reasons = bns()
    return {"reasons": reasons, **bns.batch.results(with_U=False)}


def _run_blr(st):
    bns = st["bns"]
    reasons = bns(max_iterations=st["iterations"], check=False)
    res = bns.batch.results(with_U=True)
    return {"reasons": reasons, **res, "U_sorted": res["U_sorted"].view(torch.float64)}  # this family's U is FP64


def _run_adjoint(st):
    theta = st["theta"].clone().requires_grad_(True)
    log_Z = EvidenceFn.apply(theta, st["ds"])
    log_Z.backward()
    return {"log_Z": log_Z.detach(), "grad": theta.grad}


def _run_evidence(st):
    lib, L, sender = st["lib"], st["log_L"], st["sender"]
    N = L.numel()
    e = lambda n, dt: torch.empty(n, dtype=dt, device=L.device)
    idx, counts = e(N, torch.int32), e(N, torch.int32)
    scratch_ll, scratch_i = e(2 * (N + 1), torch.int64), e(N + 1, torch.int32)
    final, log_X, log_dZ, log_Z = e(8, torch.float64), e(N, torch.float64), e(N, torch.float64), e(N, torch.float64)
    stream = ctypes.c_void_p(torch.cuda.current_stream(L.device).cuda_stream)
    p = lambda t: ctypes.c_void_p(t.data_ptr())
    rc = lib.gbns_count_crossed_edges(p(sender), p(L), N, p(idx), p(counts), p(scratch_ll), p(scratch_i), stream)
    if rc != 0:
        raise RuntimeError(lib.gbns_last_error().decode())
    sorted_L = L[idx.long()]
    rc = lib.gbns_evidence_stats(p(sorted_L), p(counts), N, p(st["ncoef"]), st["nmax"], p(final), p(log_X), p(log_dZ),
                                 p(log_Z), stream)
    if rc != 0:
        raise RuntimeError(lib.gbns_last_error().decode())
    return {"indices": idx, "counts": counts, "final": final, "log_X": log_X, "log_dZ": log_dZ, "log_Z": log_Z}


def _run_sample(st):
    return gb.sample_evidence(st["key"], st["counts"], st["log_L"], S=st["S"])


def _run_forward(st):
    return st["batch"].forward(0, st["U"])


def _run_transform(st):
    X, density = st["model"].transform_device(st["U"], log_L=st["log_L"])
    return {"X": X, "density": density}


# ------------------------------------------------------------------------- work

def _sampler_work(D, n, S, iterations, kind, N=0):
    """Likelihood evaluations of `iterations` shells of n / 2 chains at about six per slice, and the
    store they leave."""
    evals = iterations * (n // 2) * S * 6
    per = 2 * N * D if kind == "blr" else (10 * D + 22 if kind == "shells" else D * D + 8 * D)
    return evals * per, iterations * (n // 2) * 13 + n * D * 8


def work(case):
    k = case["kind"]
    if k == "call":
        D = case["D"]
        f, b = _sampler_work(D, case["live"] or 30 * D, case["slices"] or 5 * D, 12 + 4 * D, case["family"])
    elif k == "batch":
        f = b = 0
        for D in _mixed_dims(case):
            one = _sampler_work(D, case["live"] or 50 * D, case["slices"] or 5 * D, case["iterations"] or 12 + 3 * D,
                                case["family"])
            f, b = f + one[0], b + one[1]
    elif k == "blr":
        f = b = 0
        for N, P in _blr_dims(case):
            one = _sampler_work(P, case["live"] or 25 * P, 5 * P, case["iterations"], "blr", N)
            f, b = f + one[0], b + one[1] + 4 * N * (P + 1)
    elif k == "adjoint":
        M, N, P = case["M"], case["N"], case["P"]
        f, b = 2 * (2 * M * N * P + 4 * M * N), 2 * (8 * M * (P + 1) + 4 * N * (P + 1))
    elif k == "evidence":
        f, b = 60 * case["N"], 44 * case["N"]
    elif k == "sample":
        f, b = 400 * case["M"] * case["S"], 12 * case["M"] + 8 * case["S"]
    elif k == "forward":
        D, B = case["D"], case["B"]
        per = 2 * case["N"] * D if case["N"] else (10 * D + 22 if case["family"] == "shells" else D * D + 8 * D)
        f, b = B * per, B * (4 * D * (2 if case["N"] else 1) + 4)
    else:
        D, rows = case["D"], case["rows"]
        f = rows * (60 * D + (D * D if case["tril"] else 0))
        b = rows * (D * (8 + (8 if case["double"] else 4)) + 16)
    return {"bytes": float(b), "flops": float(f)}


# ------------------------------------------------------------------------- exact

def exact(case, seed):
    f = globals().get("_exact_" + case["kind"])
    return None if f is None else f(case, seed)


def _ndtri64(U):
    """The standard normal quantile in FP64: torch's, refined by two Newton steps in the nearer tail."""
    low = U <= 0.5
    tail = torch.where(low, U, 1.0 - U)
    z = torch.special.ndtri(tail)
    for _ in range(2):
        z = z - (torch.special.ndtr(z) - tail) / (torch.exp(-0.5 * z * z) / math.sqrt(2.0 * math.pi))
    return torch.where(low, z, -z)


def _exact_adjoint(case, seed):
    if case["M"] * case["N"] * case["P"] > 2e11:
        return None
    st = _prepare_adjoint(case, seed)
    ds, (log_tau, log_sigma) = st["ds"], st["theta"].tolist()
    tau, s2, N = math.exp(log_tau), math.exp(2.0 * log_sigma), case["N"]
    Phi, y = ds.Phi.double(), ds.y.double()
    ss, rp = [], []
    for i in range(0, case["M"], 4096):
        Pw = (tau * _ndtri64(ds.U[i:i + 4096])) @ Phi.T
        r = y - Pw
        ss.append((r * r).sum(1))
        rp.append((r * Pw).sum(1))
    ss, rp = torch.cat(ss), torch.cat(rp)
    a = -0.5 * N * (math.log(2.0 * math.pi) + 2.0 * log_sigma) - 0.5 * ss / s2 + ds.log_w
    p = torch.softmax(a, 0)
    return {"log_Z": torch.logsumexp(a, 0), "grad": torch.stack([(p * rp).sum() / s2, (p * (ss / s2 - N)).sum()])}


def _exact_evidence(case, seed):
    log_L, sender, _ = _sample_set(case, seed)
    N = len(log_L)
    key = np.concatenate([[-np.inf], log_L])
    order = np.argsort(key, kind="stable")
    degree = np.bincount(np.maximum(sender, 0), minlength=N + 1)
    crossed = 1 + np.cumsum(degree[order] - 1)
    L = torch.as_tensor(key[order][1:], dtype=torch.float64, device=DEVICE)
    n = torch.as_tensor(crossed[:N], dtype=torch.float64, device=DEVICE)
    ln, ln1, ln2 = torch.log(n), torch.log(n + 1.0), torch.log(n + 2.0)
    T, t = -torch.log1p(1.0 / n), -ln1
    T2, t2, tT = -torch.log1p(2.0 / n), math.log(2.0) - ln1 - ln2, -torch.log1p(1.0 / n) - ln2
    zero = torch.zeros(1, dtype=torch.float64, device=DEVICE)
    X, X2 = torch.cumsum(T, 0), torch.cumsum(T2, 0)
    Xp, X2p = torch.cat([zero, X[:-1]]), torch.cat([zero, X2[:-1]])
    mid = torch.logaddexp(L, torch.cat([zero - math.inf, L[:-1]])) - math.log(2.0)
    dZ = Xp + t + mid
    A = torch.logcumsumexp(X2p + tT + mid - X, 0)
    Ap = torch.cat([zero - math.inf, A[:-1]])
    dZ2 = X2p + t2 + 2.0 * mid
    lse = lambda v: torch.logsumexp(v, 0)
    final = torch.stack([L[-1], X[-1], X2[-1], lse(dZ), X[-1] + A[-1],
                         lse(torch.cat([math.log(2.0) + dZ + Ap, dZ2])), dZ[-1], lse(dZ2)])
    return {"indices": None, "counts": None, "final": final, "log_X": X, "log_dZ": dZ,
            "log_Z": torch.logcumsumexp(dZ, 0)}


def _threefry(k0, k1, c1):
    """Threefry-2x32-20 of the counters (0, c1) under the keys (k0, k1), int64 tensors of 32-bit words."""
    mask = 0xFFFFFFFF
    ks = (k0, k1, k0 ^ k1 ^ 0x1BD11BDA)
    x0, x1 = ks[0] + 0 * c1, (c1 + ks[1]) & mask
    rot = ((13, 15, 26, 6), (17, 29, 16, 24))
    for block in range(5):
        for r in rot[block & 1]:
            x0 = (x0 + x1) & mask
            x1 = ((x1 << r) | (x1 >> (32 - r))) & mask
            x1 = x1 ^ x0
        x0 = (x0 + ks[(block + 1) % 3]) & mask
        x1 = (x1 + ks[(block + 2) % 3] + block + 1) & mask
    return x0, x1


def _exact_sample(case, seed):
    counts, log_L = _simulated_run(case, seed)
    n = torch.as_tensor(counts, dtype=torch.float64, device=DEVICE)
    L = torch.as_tensor(log_L, device=DEVICE)
    i64 = lambda v: torch.as_tensor(v, dtype=torch.int64, device=DEVICE)
    k0, k1 = (i64(int(v)) for v in ((int(seed) >> 32) & 0xFFFFFFFF, int(seed) & 0xFFFFFFFF))
    i, out = torch.arange(len(log_L), device=DEVICE), []
    for s in range(case["S"]):
        a, b = _threefry(k0, k1, i64(s))
        c, d = _threefry(a, b, i)
        hi, lo = _threefry(c, d, 0 * i)
        u = ((hi << 20) | (lo >> 12)).double() * 2.0 ** -52
        lt = torch.log(u) / n
        X = torch.cumsum(lt, 0)
        out.append(torch.logsumexp(X - lt + torch.log(-torch.expm1(lt)) + L, 0))
    return torch.stack(out)


def _exact_forward(case, seed):
    g = _generator(seed, 6)
    U = _prepare_points64(case, seed)
    if case["family"] == "lingauss":
        model, Phi, y = _blr_problem(g, case["N"], case["D"], 0.5, 1.0)
        Phi, y = (torch.as_tensor(v, dtype=torch.float64, device=DEVICE) for v in (Phi, y))
        out = [((y - _ndtri64(U[i:i + 2048]) @ Phi.T) ** 2).sum(1) for i in range(0, len(U), 2048)]
        return -0.5 * torch.cat(out) / 0.25 - 0.5 * case["N"] * math.log(2.0 * math.pi * 0.25)
    like = _model(case["family"], case["D"], g).log_likelihood
    dev = lambda x: torch.as_tensor(x, dtype=torch.float64, device=DEVICE)
    if case["family"] == "mvn":
        L = dev(np.linalg.cholesky(like.cov))
        z = torch.linalg.solve_triangular(L, (-10.0 + 20.0 * U - dev(like.mu)).T, upper=False)
        return -0.5 * (z * z).sum(0) - torch.log(torch.diag(L)).sum() - 0.5 * case["D"] * math.log(2.0 * math.pi)
    X = -6.0 + 12.0 * U
    s = [-0.5 * ((torch.linalg.vector_norm(X - dev(c), dim=1) - 2.0) / 0.1) ** 2 for c in (like.c1, like.c2)]
    return torch.logaddexp(s[0], s[1]) - 0.5 * math.log(2.0 * math.pi * 0.01)


def _prepare_points64(case, seed):
    return _points(seed, case["B"], case["D"], torch.float64 if case["family"] == "lingauss" else torch.float32).double()


def _exact_transform(case, seed):
    g = _generator(seed, 7)
    st = _prepare_transform(case, seed)
    U, D, half = st["U"].double(), case["D"], case["D"] // 2
    dev = lambda x: torch.as_tensor(x, dtype=torch.float64, device=DEVICE)
    log_norm = 0.5 * math.log(2.0 * math.pi)
    if case["tril"]:
        loc = dev(g.standard_normal(D))
        L = dev(np.linalg.cholesky(_cov(g, D)))
        z = _ndtri64(U)
        X = loc + z @ L.T
        lp = (-0.5 * z * z - log_norm).sum(1) - torch.log(torch.diag(L)).sum()
    else:
        z = _ndtri64(U[:, half:])
        X = torch.cat([-3.0 + 8.0 * U[:, :half], 1.0 + 2.0 * z], 1)
        lp = (-0.5 * z * z - log_norm - math.log(2.0)).sum(1) - half * math.log(8.0)
    return {"X": X, "density": st["log_L"] + lp}
