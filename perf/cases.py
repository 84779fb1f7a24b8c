"""Performance cases of the GB300 SAOM simulator, through its public entry points.

Each case stands for a call that a user's program makes: a forward simulation,
a Robbins-Monro round of an estimator, the statistics of simulated end
networks, a step of the moment surrogate. The sizes are those of the
repository's own workloads (cusna_gb300/workloads.py, bench.py) or between
them. `prepare` makes seeded synthetic inputs, and whatever handle a program
keeps from call to call (a replayable plan, a network's weights).
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from cusna_gb300 import data as D
from cusna_gb300 import effects as E
from cusna_gb300 import fran as F
from cusna_gb300 import sim
from cusna_gb300 import workloads as WL
from cusna_gb300.abi import adam_hyper_bytes, check, load_library
from cusna_gb300.glue import MultiInputs, marshal_multi, marshal_period
from cusna_gb300.surrogate import MlpSurrogate

# The library times its candidate launch shapes over the first calls of a
# signature and keeps the fastest; a program that simulates in earnest makes
# hundreds of calls, so the shape is settled before a case is measured.
SETTLE = 11
_settled = set()

STRUCTURAL_EFFECTS = ("density", "recip", "transTrip", "cycle3", "transTies", "transRecTrip",
                      "inPopSqrt", "outPop", "inAct", "outActSqrt", "outTrunc", "reciAct",
                      "gwesp", "gwespFB", "gwdspFF")
STRUCTURAL_THETA = (-1.6, 1.1, 0.15, -0.1, 0.2, -0.1, 0.15, -0.05, -0.03, -0.05, 0.1, -0.05,
                    0.2, 0.1, -0.05)
STATS_EFFECTS = ("density", "recip", "transTrip", "inPopSqrt", "outAct", "outTrunc", "egoX",
                 "altX", "simX", "gwesp", "gwdspFF")
GOF_LEVELS = ((0, 1, 2, 3, 4, 5, 6, 7, 8), (0, 1, 2, 3, 4, 5, 6, 7, 8), (1, 2, 3, 4, 5, 6, 7))


def listed():
    return [
        # the smallest call: one chain of a classroom-sized period through the
        # reference-facing entry point, host buffers in and out
        dict(name="one_chain", kind="one", n=50, m=1),
        # one call of the FRAN backend that an external Robbins-Monro driver
        # makes per iteration: one chain of each of two periods
        dict(name="fran_call", kind="fran", n=50, m=1),
        # a phase-2 Robbins-Monro round of the estimator: a replayed plan of two
        # periods, statistics only (the bench's n=300 panel)
        dict(name="phase2_round", kind="phase2", n=300, m=256),
        # forward simulation at fixed parameters with scores, host buffers (the
        # bench's headline workload)
        dict(name="forward", kind="forward", n=200, m=4096),
        # the largest: network-behaviour co-evolution (the bench's n=1000 workload)
        dict(name="coevolution", kind="coevol", n=1000, m=1024),
        # uneven groups in one conditional round, n ~ U{20..400}, one chain each
        dict(name="groups_round", kind="groups", n=400, m=256),
        # two co-evolving networks with every cross-network effect, end networks out
        dict(name="multi_network", kind="multi", n=200, m=1024),
        # a model with many structural and weighted-shared-partner effects, odd n
        dict(name="structural", kind="structural", n=129, m=512),
        # statistics of simulated end networks (targets, goodness of fit)
        dict(name="end_stats", kind="stats", n=100, m=1000),
        # sienaGOF's three auxiliary distributions of simulated end networks
        dict(name="gof", kind="gof", n=100, m=1000),
        # an epoch of the moment surrogate's training (batches of 1024)
        dict(name="surrogate_epoch", kind="train", n=12, m=1024),
        # the surrogate's mean and Jacobian at one parameter point, two periods:
        # one iteration of phases 1-2 on the surrogate
        dict(name="surrogate_point", kind="point", n=8, m=2),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["one", "fran", "phase2", "forward", "coevol", "groups", "multi",
                       "structural", "stats", "gof", "train", "point"])
    if kind == "one":
        n, m = _log_int(rng, 20, 130), _log_int(rng, 1, 8)
    elif kind == "fran":
        n, m = _log_int(rng, 25, 130), 1
    elif kind == "phase2":
        n, m = _log_int(rng, 40, 400), _log_int(rng, 32, 512)
    elif kind == "forward":
        n = _log_int(rng, 30, 400)
        m = _log_int(rng, 64, max(65, min(4096, int(1.6e8 / (n * n)))))
    elif kind == "coevol":
        n = _log_int(rng, 60, 1000)
        m = _log_int(rng, 64, min(1024, int(1e9 / (n * n))))
    elif kind == "groups":
        n, m = rng.randint(100, 400), _log_int(rng, 16, 256)
    elif kind == "multi":
        n, m = _log_int(rng, 30, 260), _log_int(rng, 32, 512)
    elif kind == "structural":
        n, m = _log_int(rng, 30, 260), _log_int(rng, 32, 256)
    elif kind == "stats":
        n, m = _log_int(rng, 20, 260), _log_int(rng, 1, 1000)
    elif kind == "gof":
        n, m = _log_int(rng, 20, 200), _log_int(rng, 8, 1000)
    elif kind == "train":
        n, m = rng.randint(1, 16), 16 * rng.randint(8, 128)
    else:
        n, m = rng.randint(1, 12), _log_int(rng, 1, 64)
    return dict(kind=kind, n=n, m=m)


# ---- seeded inputs ------------------------------------------------------------
def _rng(seed):
    return np.random.Generator(np.random.PCG64(int(seed)))


def _net(r, n, p):
    a = (r.random((n, n)) < p).astype(np.uint8)
    np.fill_diagonal(a, 0)
    return a


def _cov(r, n):
    return r.standard_normal(n).astype(np.float32).astype(np.float64)


def _density(n):
    """Mean outdegree 6 as the synthetic panels have it (0.03 at n = 200), less
    in the smallest networks."""
    return min(6.0 / max(n - 1, 1), 0.12)


def _next_wave(r, x):
    """A wave some dyads away from x: a fifth of its ties end, as many begin."""
    n = x.shape[0]
    keep = r.random((n, n)) < 0.8
    new = r.random((n, n)) < 0.2 * x.mean()
    y = ((x != 0) & keep) | ((x == 0) & new)
    np.fill_diagonal(y, False)
    return y.astype(np.int64)


def _fran_inputs(case, seed):
    r = _rng(seed)
    n = case["n"]
    waves = [_net(r, n, _density(n)).astype(np.int64)]
    for _ in range(2):
        waves.append(_next_wave(r, waves[-1]))
    return waves, np.array([-2.4, 1.9, 0.3]) + 0.02 * r.standard_normal(3), int(r.integers(1, 2**31))


def _one_inputs(case, seed):
    r = _rng(seed)
    n = case["n"]
    x0 = _net(r, n, _density(n))
    theta = np.array([-2.5, 2.0, 0.3]) + 0.02 * r.standard_normal(3)
    return x0, theta, 6.0, int(r.integers(1, 2**62))


def _stats_inputs(case, seed):
    r = _rng(seed)
    n, m = case["n"], case["m"]
    a = (r.random((m, n, n)) < _density(n)).astype(np.uint8)
    a[:, np.arange(n), np.arange(n)] = 0
    return a, _cov(r, n)


def _effects(names, cov=None):
    return [E.make_effect_spec(nm, cov if nm in E.COVARIATE else None) for nm in names]


def _period(case, seed):
    """The marshalled call of a single-network case and its repeatable inputs."""
    kind, n, m = case["kind"], case["n"], case["m"]
    if kind == "one":
        x0, theta, lam, key = _one_inputs(case, seed)
        inp = WL.period_inputs(x0, _effects(WL.C3_EFFECTS[:3]))
        return marshal_period(inp, m, key, lam, theta)
    r = _rng(seed)
    x0 = _net(r, n, _density(n))
    key = int(r.integers(1, 2**62))
    if kind == "forward":
        inp = WL.period_inputs(x0, _effects(WL.C2_EFFECTS, _cov(r, n)))
        theta = WL.C2_THETA + 0.01 * r.standard_normal(len(WL.C2_THETA))
        return marshal_period(inp, m, key, 8.0, theta)
    if kind == "structural":
        inp = WL.period_inputs(x0, _effects(STRUCTURAL_EFFECTS))
        theta = np.array(STRUCTURAL_THETA) * (1.0 + 0.02 * r.standard_normal(len(STRUCTURAL_THETA)))
        return marshal_period(inp, m, key, 5.0, theta)
    z = r.integers(1, 6, size=n).astype(np.float64)   # coevol
    beh = D.build_behavior_data(np.stack([z, z], axis=1), n, 2)
    effs = _effects(("density", "recip", "transTrip"))
    effs += [E.make_effect_spec(nm, dyn=True) for nm in ("egoX", "altX", "simX")]
    bef = [E.make_beh_effect_spec(nm) for nm in ("linear", "quad", "avAlt")]
    inp = WL.period_inputs(x0, effs, 1, beh, D.beh_values_less_missing_starts(beh, 1), bef)
    theta = WL.C4_THETA + 0.01 * r.standard_normal(len(WL.C4_THETA))
    return marshal_period(inp, m, key, 4.0, theta, lamb=2.0, thetab=WL.C4_THETAB)


def _plan(case, seed):
    """A replayable plan's problems and the parameter rows of the next round."""
    kind, n, m = case["kind"], case["n"], case["m"]
    r = _rng(seed)
    ms = []
    if kind == "phase2":
        cov = _cov(r, n)
        theta = WL.C5_THETA + 0.01 * r.standard_normal(len(WL.C5_THETA))
        for _ in range(2):
            inp = WL.period_inputs(_net(r, n, _density(n)), WL.c5_effects(cov))
            p = marshal_period(inp, m, int(r.integers(1, 2**31)), WL.C5_LAMBDA, theta)
            p.drop_outputs(("scores",))
            ms.append(p)
        return ms, dict(theta=theta.astype(np.float32)[None, :],
                        lam=np.full((2, 1), WL.C5_LAMBDA, np.float32))
    theta = WL.C3_THETA + 0.01 * r.standard_normal(len(WL.C3_THETA))
    for _ in range(m):
        g = int(r.integers(20, n + 1))
        x0 = _net(r, g, float(r.uniform(0.02, 0.10)))
        cov = (r.random(g) < 0.5).astype(np.float64)
        inp = WL.period_inputs(x0, WL.c3_effects(cov), conditional=1, target_dist=3 * g // 2)
        ms.append(marshal_period(inp, 1, int(r.integers(1, 2**31)), 1.0, theta))
    return ms, dict(theta=theta.astype(np.float32)[None, :])


def _multi(case, seed):
    r = _rng(seed)
    n, m = case["n"], case["m"]
    p = min(0.06, 12.0 / n)
    x0s = [_net(r, n, p), _net(r, n, 1.3 * p)]
    effs, theta = [], []
    for d in range(2):
        for name, t in (("density", -2.0), ("recip", 0.9), ("transTrip", 0.15), ("crprod", 0.6),
                        ("crprodRecip", 0.3), ("crprodMutual", -0.2), ("from", 0.1), ("to", 0.05)):
            effs.append(E.make_effect_spec(name, net_ref=1 - d if name in E.CROSSNET else None))
            theta.append(t)
    pe = E.prepare_effects_v2(effs, n, 1, None, None)
    inp = MultiInputs(x0s=x0s, type_ids=np.asarray(pe.type_ids, np.int32),
                      netof=np.repeat(np.arange(2), len(effs) // 2).astype(np.int32),
                      netref=E.effect_netrefs(effs), etypes=E.effect_etypes(effs),
                      wtab=E.effect_wtabs(effs, n), p1=pe.p1, p2=pe.p2, vmat=pe.vmat,
                      symf=np.zeros(2, np.int32))
    return marshal_multi(inp, m, int(r.integers(1, 2**62)), np.array([3.8, 4.9]), np.array(theta))


def _mlp_params(r, n_in, h, n_out, scale):
    """Weights and biases of a network some epochs into its training."""
    return [r.standard_normal((h, n_in)) * math.sqrt(2 / n_in), scale * r.standard_normal(h),
            r.standard_normal((h, h)) * math.sqrt(2 / h), scale * r.standard_normal(h),
            scale * r.standard_normal((n_out, h)), scale * r.standard_normal(n_out)]


def _train_inputs(case, seed):
    """Pairs, row order, weights and Adam moments of an epoch in mid-training."""
    steps, batch = case["n"], case["m"]
    r = _rng(seed)
    n_in, h, n_out, rows = 16, 256, 8, steps * batch
    flat = np.concatenate([x.ravel() for x in _mlp_params(r, n_in, h, n_out, 0.05)])
    x = r.standard_normal((rows, n_in))
    t = np.tanh(x[:, :n_out]) + 0.3 * x[:, n_out:2 * n_out] * x[:, :n_out] \
        + 0.1 * r.standard_normal((rows, n_out))
    arrs = dict(params=flat, m=1e-3 * r.standard_normal(flat.size),
                v=np.exp(r.uniform(-10.0, -6.0, flat.size)), x=x, t=t)
    arrs = {k: v.astype(np.float32) for k, v in arrs.items()}
    return arrs, r.permutation(rows).astype(np.int32)


TRAIN_STEP0, TRAIN_LR = 400, 1e-3


def _point_inputs(case, seed):
    r = _rng(seed)
    params = np.concatenate([x.ravel() for x in _mlp_params(r, 16, 256, 8, 0.1)]).astype(np.float32)
    return r.standard_normal((case["m"], 16)).astype(np.float32).astype(np.float64), params


# ---- prepare and run ----------------------------------------------------------
def _settle(case, call):
    key = (case["kind"], case["n"], case["m"])
    if key not in _settled:
        for _ in range(SETTLE):
            call()
        _settled.add(key)


def prepare(case, seed):
    # a program that will make many calls asks for the specialised kernels at once
    sim.specialise_mode(2)
    kind = case["kind"]
    if kind in ("one", "forward", "coevol", "structural"):
        m = _period(case, seed)
        _settle(case, lambda: sim.simulate(m))
        return dict(kind=kind, m=m)
    if kind == "multi":
        m = _multi(case, seed)
        _settle(case, lambda: sim.simulate_multi(m))
        return dict(kind=kind, m=m)
    if kind in ("phase2", "groups"):
        ms, rows = _plan(case, seed)
        plan = sim.SimPlan(ms)
        for _ in range(SETTLE):    # a plan settles its own launch shape
            plan.launch()
        plan.set_epoch(0)
        return dict(kind=kind, plan=plan, rows=rows)
    if kind == "fran":
        waves, theta, s = _fran_inputs(case, seed)
        return dict(kind=kind, theta=theta, fran=F.cusna_fran(waves, WL.C3_EFFECTS[:3], seed=s))
    if kind == "stats":
        a, cov = _stats_inputs(case, seed)
        effs = _effects(STATS_EFFECTS, cov)
        pe = E.prepare_effects_v2(effs, case["n"])
        args = (case["n"], len(effs), pe.type_ids, pe.p1, pe.p2, pe.vmat, None, None, None, None,
                None, E.effect_wtabs(effs, case["n"]), 0)
        return dict(kind=kind, a=a, args=args)
    if kind == "gof":
        return dict(kind=kind, a=_stats_inputs(case, seed)[0])
    lib = load_library()
    if kind == "train":
        arrs, order = _train_inputs(case, seed)
        s = {k: torch.from_numpy(v).cuda() for k, v in arrs.items()}
        wb = int(lib.cusna_mlp_workspace_bytes(16, 256, 8, case["m"]))
        s.update(kind=kind, lib=lib, batch=case["m"], steps=case["n"], wb=wb,
                 rows=torch.from_numpy(order).cuda(), grad=torch.zeros_like(s["params"]),
                 hyper=torch.from_numpy(adam_hyper_bytes(TRAIN_STEP0, TRAIN_LR)).cuda(),
                 losses=torch.zeros(case["n"], device="cuda"),
                 work=torch.empty(wb, dtype=torch.uint8, device="cuda"))
        return s
    X, params = _point_inputs(case, seed)   # point
    net = MlpSurrogate(16, 8, 256, seed=1)
    net.load_params(params)
    return dict(kind=kind, net=net, X=X, n_wrt=case["n"])


def run(state):
    kind = state["kind"]
    if kind in ("one", "forward", "coevol", "structural"):
        return dict(sim.simulate(state["m"]))
    if kind == "multi":
        return dict(sim.simulate_multi(state["m"]))
    if kind in ("phase2", "groups"):
        plan = state["plan"]
        plan.set_params(**state["rows"])
        plan.launch()
        outs = plan.outputs()
        return {k: np.concatenate([o[k] for o in outs]) for k in outs[0]}
    if kind == "fran":
        got = state["fran"]({"theta": state["theta"]})
        return [got["fra"], got["sc"], got["ntim0"]]
    if kind == "stats":
        return sim.network_stats(state["a"], *state["args"])
    if kind == "gof":
        return [sim.gof_distribution(state["a"], q, lv) for q, lv in enumerate(GOF_LEVELS)]
    if kind == "train":
        lib, s = state["lib"], state
        check(lib.cusna_mlp_train_steps(
            s["params"].data_ptr(), s["grad"].data_ptr(), s["m"].data_ptr(), s["v"].data_ptr(),
            s["x"].data_ptr(), s["t"].data_ptr(), s["rows"].data_ptr(), s["batch"], s["steps"],
            s["hyper"].data_ptr(), s["losses"].data_ptr(), s["work"].data_ptr(),
            C.c_size_t(s["wb"]), 16, 256, 8, 1, torch.cuda.current_stream().cuda_stream),
            "cusna_mlp_train_steps", lib)
        return [s["params"], s["m"], s["v"], s["losses"]]
    return list(state["net"].predict_with_jacobian(state["X"], state["n_wrt"]))


# ---- the work a pass cannot do without ------------------------------------------
def _sim_work(n, k, m, lam, pairs, scores=True, deg=6.0):
    """m chains of a period: n * lam ministeps of n alters. Per alter: the
    Philox block (10 rounds of 6 operations), the Gumbel transform (two
    logarithms), the k-term predictor, with scores its exponential and the
    k + 1 sums, and a table entry or count per effect; the two-path counts of a
    ministep cost `pairs` passes over the focal actor's neighbourhood's rows."""
    steps = m * n * lam
    per_alter = 60 + 10 + 3 * k + ((10 + 2 * (k + 1)) if scores else 0)
    flops = steps * (n * per_alter + pairs * deg * n / 32)
    return flops, m * (8 * k + 4 * (k + 1) * scores + 24) + n * n / 4


def work(case):
    kind, n, m = case["kind"], case["n"], case["m"]
    if kind == "one":
        flops, byts = _sim_work(n, 3, m, 6.0, 2)
    elif kind == "fran":
        flops, byts = _sim_work(n, 3, 2, 2.0, 2)
    elif kind == "phase2":
        flops, byts = _sim_work(n, 7, 2 * m, 7.0, 3, scores=False)
    elif kind == "forward":
        flops, byts = _sim_work(n, 8, m, 8.0, 3)
    elif kind == "structural":
        flops, byts = _sim_work(n, len(STRUCTURAL_EFFECTS), m, 5.0, 8)
    elif kind == "coevol":
        flops, byts = _sim_work(n, 6, m, 4.0, 2)
        byts += 4.0 * n * m
    elif kind == "groups":
        mean_n2 = (n * n + 20 * n + 400) / 3.0
        flops, byts = _sim_work(math.sqrt(mean_n2), 4, m, 2.0, 2, deg=13.0)
    elif kind == "multi":
        flops, byts = _sim_work(n, 8, 2 * m, 4.35, 4, deg=12.0)
        byts += 2.0 * m * n * n
    elif kind == "stats":
        ties = n * n * _density(n)
        flops = m * (ties * 12 + n * n * _density(n) * n * 0.2 + n * n)
        byts = float(m) * n * n + 8.0 * m * len(STATS_EFFECTS)
    elif kind == "gof":
        flops = m * (n * n * math.ceil(n / 32) * 1.0 + 2.0 * n * n)
        byts = float(m) * n * n + 8.0 * m * sum(len(v) for v in GOF_LEVELS)
    elif kind == "train":
        per_row = 16 * 256 + 256 * 256 + 256 * 8
        npar = per_row + 256 + 256 + 8
        flops = n * (6.0 * m * per_row - 2.0 * m * 16 * 256 + 12.0 * npar)
        byts = n * (m * 24 * 4.0) + 6.0 * 4 * npar
    else:
        per_row = 16 * 256 + 256 * 256 + 256 * 8
        flops = 2.0 * m * per_row + 2.0 * m * n * (256 * 256 + 256 * 8 + 256)
        byts = 4.0 * per_row + 4.0 * m * (16 + 8 + 8 * n)
    return {"bytes": float(byts), "flops": float(flops)}


# ---- plain 64-bit values ------------------------------------------------------------
def _philox(c0, c1, c2, c3, key):
    """Philox4x32-10 of arrays of counters (Salmon et al. 2011)."""
    c = [np.asarray(v, dtype=np.uint64) & 0xFFFFFFFF for v in np.broadcast_arrays(c0, c1, c2, c3)]
    k0, k1 = key & 0xFFFFFFFF, key >> 32 & 0xFFFFFFFF
    low, s32 = np.uint64(0xFFFFFFFF), np.uint64(32)
    for _ in range(10):
        p0, p1 = c[0] * np.uint64(0xD2511F53), c[2] * np.uint64(0xCD9E8D57)
        c = [(p1 >> s32) ^ c[1] ^ np.uint64(k0), p1 & low, (p0 >> s32) ^ c[3] ^ np.uint64(k1), p0 & low]
        k0, k1 = (k0 + 0x9E3779B9) & 0xFFFFFFFF, (k1 + 0xBB67AE85) & 0xFFFFFFFF
    return [v.astype(np.float64) for v in c]


def _unit(x):
    return (x + 0.5) * 2.0**-32


def _exact_chain(x0, theta, lam, key, chain, target=None):
    """One chain of a density, reciprocity and transitive-triplet model."""
    n = x0.shape[0]
    th = np.asarray(theta, dtype=np.float32).astype(np.float64)
    a, x0 = x0.astype(np.float64), x0.astype(np.float64)
    js, sc, t, steps, dist = np.arange(n), np.zeros(3), 0.0, 0, 0
    while True:
        w = _philox(steps, chain, 0, 0, key)
        t += -math.log(_unit(float(w[0]))) / (n * lam)
        if target is None and t > 1.0:
            break
        i = min(int(_unit(float(w[2])) * n), n - 1)
        sign = 1.0 - 2.0 * a[i]
        d = np.stack([sign, sign * a[:, i], sign * (a[i] @ a + a @ a[i])])
        d[:, i] = 0.0
        f = th @ d
        g = f - np.log(-np.log(_unit(_philox(steps, chain, 1, js, key)[0])))
        j = int(np.argmax(g))
        e = np.exp(f - f.max())
        sc += d[:, j] - (d @ e) / e.sum()
        steps += 1
        if j != i:
            dist += 1 if a[i, j] == x0[i, j] else -1
            a[i, j] = 1.0 - a[i, j]
        if target is not None and dist >= target:
            break
    stats = np.array([a.sum(), (a * a.T).sum(), (a * (a @ a)).sum()])
    return dict(stats=stats, scores=np.concatenate([[steps / lam - n], sc]), ntim=t, dist=dist,
                dist_stat=int((a != x0).sum()), steps=steps)


def _exact_sim(case, seed):
    if case["kind"] == "one":
        x0, theta, lam, key = _one_inputs(case, seed)
        got = [_exact_chain(x0, theta, lam, key, c) for c in range(case["m"])]
        return {k: np.array([g[k] for g in got]) for k in got[0]}
    waves, theta, s = _fran_inputs(case, seed)
    r = _rng(s)
    fra, sc, nt = [], [], []
    for q in range(2):
        target = int((waves[q + 1] != waves[q]).sum())
        got = _exact_chain(waves[q], theta, 1.0, int(r.integers(1, np.iinfo(np.int32).max)), 0, target)
        fra.append(got["stats"])
        sc.append(got["scores"][1:])
        nt.append(got["ntim"])
    return [np.array(fra), np.array(sc), np.array(nt)]


def _exact_stats(case, seed):
    an, cov = _stats_inputs(case, seed)
    n = case["n"]
    a = torch.from_numpy(an).cuda().double()
    v = cov - cov.mean()
    rng = cov.max() - cov.min()
    off = ~np.eye(n, dtype=bool)
    dist = np.abs(cov[:, None] - cov[None, :])
    simm = float((1.0 - dist[off] / rng).mean())
    vt = torch.from_numpy(v).cuda()
    sx = torch.from_numpy(1.0 - dist / rng - simm).cuda()
    od, idg = a.sum(2), a.sum(1)
    aa, at = a @ a, a @ a.transpose(1, 2)
    ea = math.exp(0.69)

    def gw(c):
        return ea * (1.0 - (1.0 - math.exp(-0.69)) ** c)
    offt = torch.from_numpy(off).cuda().double()
    cols = [a.sum((1, 2)), (a * a.transpose(1, 2)).sum((1, 2)), (a * aa).sum((1, 2)),
            (idg ** 1.5).sum(1), (od * od).sum(1), torch.clamp(od, max=1.0).sum(1), od @ vt, idg @ vt,
            (a * sx).sum((1, 2)), (a * gw(aa)).sum((1, 2)), (gw(aa) * offt).sum((1, 2))]
    del at
    return torch.stack(cols, 1).cpu().numpy()


def _exact_gof(case, seed):
    a = torch.from_numpy(_stats_inputs(case, seed)[0]).cuda().double()
    n = case["n"]
    out = [torch.stack([(a.sum(1 + q) <= lv).double().sum(1) for lv in GOF_LEVELS[q]], 1)
           for q in range(2)]
    reach = a.clone()
    eye = torch.eye(n, dtype=torch.float64, device="cuda")
    cols = []
    for _ in GOF_LEVELS[2]:
        cols.append((reach * (1 - eye)).sum((1, 2)))
        reach = ((reach + reach @ a) > 0).double()
    out.append(torch.stack(cols + [n * (n - 1.0) - cols[-1]], 1))
    return [x.cpu().numpy() for x in out]


def _split(p, n_in=16, h=256, n_out=8):
    out, o = [], 0
    for shape in ((h, n_in), (h,), (h, h), (h,), (n_out, h), (n_out,)):
        c = math.prod(shape)
        out.append(p[o:o + c].reshape(shape))
        o += c
    return out


def _mlp64(p, x):
    w1, b1, w2, b2, w3, b3 = _split(p)
    gelu = torch.nn.functional.gelu
    return gelu(gelu(x @ w1.T + b1) @ w2.T + b2) @ w3.T + b3


def _exact_train(case, seed):
    arrs, order = _train_inputs(case, seed)
    s = {k: torch.from_numpy(v).cuda().double() for k, v in arrs.items()}
    b1, b2, eps, losses = 0.9, 0.999, 1e-8, []
    rows = torch.from_numpy(order.astype(np.int64)).cuda()
    for q in range(case["n"]):
        sel = rows[q * case["m"]:(q + 1) * case["m"]]
        p = s["params"].clone().requires_grad_(True)
        loss = ((_mlp64(p, s["x"][sel]) - s["t"][sel]) ** 2).mean()
        g, = torch.autograd.grad(loss, p)
        losses.append(loss.detach())
        s["m"] = b1 * s["m"] + (1 - b1) * g
        s["v"] = b2 * s["v"] + (1 - b2) * g * g
        t = TRAIN_STEP0 + q + 1
        s["params"] = s["params"] - TRAIN_LR * (s["m"] / (1 - b1 ** t)) \
            / ((s["v"] / (1 - b2 ** t)).sqrt() + eps)
    return [s["params"], s["m"], s["v"], torch.stack(losses)]


def _exact_point(case, seed):
    X, params = _point_inputs(case, seed)
    p, x = torch.from_numpy(params).double(), torch.from_numpy(X)
    J = torch.func.vmap(torch.func.jacrev(lambda r: _mlp64(p, r)))(x)
    return [_mlp64(p, x).numpy(), J[:, :, :case["n"]].contiguous().numpy()]


def exact(case, seed):
    """Values of the cases that a plain 64-bit restatement reaches in seconds; a
    batch of thousands of chains it does not."""
    kind = case["kind"]
    if kind in ("one", "fran"):
        return _exact_sim(case, seed)
    if kind == "stats":
        return _exact_stats(case, seed)
    if kind == "gof":
        return _exact_gof(case, seed)
    if kind == "train":
        return _exact_train(case, seed)
    if kind == "point":
        return _exact_point(case, seed)
    return None
