"""The workloads this engine is timed on, each through its public entry points.

A case is a dict of plain values with a "kind":

  iterate   one weight iteration with host buffers (Engine.iterate_host): the
            weights go in, therm + nup attempts per chain run, the weight
            update follows, and the weights, the histogram and its summary
            come back -- the loop body of a program that keeps the weights on
            the host
  run       a whole device-driven weight estimation (Engine.weight_run) from
            the zero weight, K iterations per CUDA graph, with the first
            `iters` iterations of the reference schedule
  produce   one Delta point of the production program: weights in, shift,
            thermalisation sweep, recorded sweep into the 2D (E_Delta, M)
            histogram, reweighted observables
  random    one iteration of the random-site algorithm of the CPU program
            (muca_mag): sweep, CPU-flavour update, weights and histogram out
  batch     many uneven instances at once (Batch): initial weights in, a run
            of `iters` iterations, weights out
  train     a stretch of Adam steps of the warm-start network, losses and
            parameters out
  reweight  the reweighting sums of a 2D histogram in device memory at a few
            Delta points (observables_noalloc)

Weights have the shape of a converged multicanonical weight at T = 0.5 (a
drift of some 4 units of lnW per bin, as found at L = 128) with the noise a
finite histogram leaves; chains start spread over all of E_Delta, as a
converged run's chains are.
"""
from __future__ import annotations

import math

import numpy as np
import torch

import muca_gb300 as m

BETA = 2.0  # T = 0.5


def listed():
    return [
        # the smallest run of the configurations (L=16, one block of chains):
        # launches, copies and the latency of a single warp
        {"name": "iterate_L16_c256", "kind": "iterate", "L": 16, "chains": 256, "rounds": 7, "rule": 0},
        # the headline workload: one iteration of the weight program
        {"name": "iterate_L72_c16384", "kind": "iterate", "L": 72, "chains": 16384, "rounds": 7, "rule": 0},
        # the weight estimation that the L=128 production starts from
        {"name": "iterate_L128_c16384", "kind": "iterate", "L": 128, "chains": 16384, "rounds": 7, "rule": 0},
        # the programs' default chain count (threads per SM times SMs), the largest
        {"name": "iterate_L72_c311296", "kind": "iterate", "L": 72, "chains": 311296, "rounds": 7, "rule": 0},
        # a lattice size that is not a multiple of 8 and a ragged chain count,
        # the ten-round generator and the recursion
        {"name": "iterate_L30_c4000_r10", "kind": "iterate", "L": 30, "chains": 4000, "rounds": 10, "rule": 2},
        # the first part of a weight run from the zero weight (NUPDATES small:
        # the width of the visited range still grows)
        {"name": "run_L32_c2048", "kind": "run", "L": 32, "chains": 2048, "iters": 128, "starting_M": 64,
         "graph_iters": 32},
        # the production configuration at its full shape, one sweep each
        {"name": "produce_L128_c16384", "kind": "produce", "L": 128, "chains": 16384, "rounds": 7},
        # a small production run with a ragged chain count and half-filled words
        {"name": "produce_L40_c1000", "kind": "produce", "L": 40, "chains": 1000, "rounds": 7},
        # the CPU program's algorithm with the host's logarithm
        {"name": "random_L72_c16384", "kind": "random", "L": 72, "chains": 16384, "host_logf": True},
        # the data generation of the warm start: uneven instances, 256 chains each
        {"name": "batch_64_instances", "kind": "batch", "instances": 64, "Lmin": 16, "Lmax": 128, "chains": 256,
         "iters": 16},
        # the warm-start network's training (its minibatch and last learning rates)
        {"name": "train_b4096", "kind": "train", "points": 663816, "batch": 4096, "steps": 64, "lr": 3e-4},
        # a Delta scan over one L=128 production histogram
        {"name": "reweight_L128", "kind": "reweight", "L": 128, "deltas": 4},
    ]


# the most attempts of a drawn case: those of the largest listed one
MAX_ATTEMPTS = 2 * 311296 * 72 * 72


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _draw_chains(rng, L, hi):
    return max(32, min(_log_int(rng, 64, hi), MAX_ATTEMPTS // (2 * L * L)))


def draw(rng):
    kind = rng.choice(["iterate", "iterate", "iterate", "run", "produce", "produce", "random", "batch", "train",
                       "reweight"])
    if kind == "iterate":
        L = 2 * _log_int(rng, 4, 64)
        hi = 311296 if L % 8 == 0 else 20000
        return {"kind": kind, "L": L, "chains": _draw_chains(rng, L, hi), "rounds": rng.choice([7, 7, 10]),
                "rule": rng.choice([0, 0, 1, 2])}
    if kind == "run":
        L = 2 * _log_int(rng, 4, 40)
        return {"kind": kind, "L": L, "chains": _log_int(rng, 64, 20000 if L % 8 == 0 else 4000),
                "iters": rng.choice([32, 64, 128]), "starting_M": rng.choice([1, 64, L * L]),
                "graph_iters": rng.choice([16, 32])}
    if kind == "produce":
        L = 2 * _log_int(rng, 4, 64)
        return {"kind": kind, "L": L, "chains": _draw_chains(rng, L, 32768 if L % 8 == 0 else 8000),
                "rounds": rng.choice([7, 7, 10])}
    if kind == "random":
        L = 2 * _log_int(rng, 4, 64)
        return {"kind": kind, "L": L, "chains": _log_int(rng, 64, 20000), "host_logf": rng.choice([True, False])}
    if kind == "batch":
        lo = 8 * rng.randint(1, 6)
        return {"kind": kind, "instances": _log_int(rng, 4, 63), "Lmin": lo, "Lmax": min(128, lo + 8 * rng.randint(0, 10)),
                "chains": _log_int(rng, 64, 1024), "iters": rng.randint(4, 16)}
    if kind == "train":
        return {"kind": kind, "points": _log_int(rng, 2000, 663816), "batch": _log_int(rng, 128, 8192),
                "steps": rng.randint(16, 96), "lr": rng.choice([3e-4, 1e-4])}
    return {"kind": kind, "L": 2 * _log_int(rng, 8, 64), "deltas": rng.randint(1, 6)}


# ---- inputs ---------------------------------------------------------------

def _weights(L, seed):
    """lnW over E_Delta = 0..N: mean-field entropy and energy at T = 0.5,
    whose concave parts a converged weight bridges by a straight line, plus
    the noise of a histogram of finite counts; lnW[0] = 0."""
    N = L * L
    x = np.arange(N + 1) / N
    with np.errstate(divide="ignore", invalid="ignore"):
        h = -np.where(x > 0, x * np.log(x), 0.0) - np.where(x < 1, (1 - x) * np.log(1 - x), 0.0)
    s = N * (0.25 * h + 4.0 * x + 0.02 * x * (x - 1.0))
    w = -s + np.random.default_rng(seed).normal(0.0, 0.03, N + 1)
    return w - w[0]


def _pinned(n, dtype):
    return torch.zeros(n, dtype=torch.float64, pin_memory=True).numpy().view(dtype)


def _prepare_iterate(c, seed):
    e = m.Engine(c["L"], nchains=c["chains"], rounds=c["rounds"])
    e.init_chains(m.INIT_GRADED, seed % 997)
    n = e.N + 1
    lnw = _pinned(n, np.float64)
    lnw[:] = _weights(c["L"], seed)
    return {"e": e, "lnw": lnw, "out": _pinned(n, np.float64), "hist": _pinned(n, np.uint64), "k": seed % 1000,
            "rule": c["rule"]}


def _run_iterate(s):
    e = s["e"]
    st = e.iterate_host(s["lnw"], s["k"], 100, 1000, e.N, e.N, s["rule"], lnw_out=s["out"], hist_out=s["hist"],
                        stats=True)
    s["k"] += 1
    return {"lnw": s["out"], "hist": s["hist"].view(np.int64), "d_kl": st.d_kl, "min_over_mean": st.min_over_mean,
            "start": st.start, "end": st.end, "visited": st.visited, "events": st.events, "min_count": st.min_count}


def _prepare_run(c, seed):
    e = m.Engine(c["L"], nchains=c["chains"])
    return {"e": e, "zero": np.zeros(e.N + 1), "jack": seed % 997, "c": c}


def _run_run(s):
    e, c = s["e"], s["c"]
    e.set_weights(s["zero"])
    res, recs = e.weight_run(starting_M=c["starting_M"], jack=s["jack"], max_iter=c["iters"], records=c["iters"],
                             graph_iters=c["graph_iters"], reinit_chains=1)
    return {"lnw": e.get_weights(), "hist": e.histogram().view(np.int64), "state": list(e.chain_state()),
            "iterations": res.iterations, "total_run": res.total_run,
            "width": np.array([r.width for r in recs], np.int64),
            "nupdates": np.array([r.nupdates for r in recs], np.int64), "d_kl": np.array([r.d_kl for r in recs])}


def _prepare_produce(c, seed):
    e = m.Engine(c["L"], nchains=c["chains"], mode=m.MODE_PRODUCE, rounds=c["rounds"])
    e.init_chains(m.INIT_GRADED, seed % 997)
    return {"e": e, "lnw": _weights(c["L"], seed), "k": seed % 1000, "delta": 1.96}


def _run_produce(s):
    e = s["e"]
    e.set_weights(s["lnw"])
    e.weight_shift(BETA, s["delta"])
    e.sweep(0, 100 + s["k"], 1000, e.N, 0)
    e.sweep(s["k"], 100, 2000, 0, e.N)
    o = e.observables(BETA, s["delta"])
    s["k"] += 1
    ej, ed, mg = e.chain_state()
    return {"m_abs": o.m_abs, "chi": o.chi, "u4": o.u4, "sum": o.sum, "m1": o.m1, "m2": o.m2, "m4": o.m4,
            "ej": ej, "edel": ed, "mag": mg}


def _prepare_random(c, seed):
    e = m.Engine(c["L"], nchains=c["chains"], algorithm=m.ALGO_RANDOM_SITE, host_logf=1 if c["host_logf"] else 0)
    e.init_chains(m.INIT_MUCA_MAG, seed % 997)
    return {"e": e, "lnw": _weights(c["L"], seed), "jack": seed % 997, "k": seed % 1000,
            "hist": np.zeros(e.N + 1, np.uint64), "out": np.zeros(e.N + 1)}


def _run_random(s):
    e = s["e"]
    e.set_weights(s["lnw"])
    e.sweep(s["k"], s["jack"], 0, 0, e.N)
    st = e.update_weights(m.UPDATE_TRIVIAL_CPU)
    s["k"] += 1
    return {"lnw": e.get_weights(s["out"]), "hist": e.histogram(s["hist"]).view(np.int64), "d_kl": st.d_kl,
            "start": st.start, "end": st.end, "state": list(e.chain_state())}


def _prepare_batch(c, seed):
    rng = np.random.default_rng(seed)
    sizes = list(range(c["Lmin"], c["Lmax"] + 1, 8))
    inst = [(sizes[i % len(sizes)], c["chains"], 1.0 / float(rng.uniform(0.4, 0.8)), i) for i in range(c["instances"])]
    b = m.Batch(inst)
    return {"b": b, "lnw": [_weights(x[0], seed + i) for i, x in enumerate(inst)], "iters": c["iters"]}


def _run_batch(s):
    b = s["b"]
    for i, w in enumerate(s["lnw"]):
        b.set_weights(i, w)
    res, _ = b.run(starting_M=1, starting_sweeps=1, max_iter=s["iters"], graph_iters=s["iters"], reinit_chains=1)
    n = len(s["lnw"])
    return {"lnw": np.concatenate([b.get_weights(i) for i in range(n)]), "d_kl": np.array([r.d_kl for r in res]),
            "width": np.array([r.width for r in res], np.int64),
            "nupdates": np.array([r.nupdates for r in res], np.int64),
            "total_run": np.array([r.total_run for r in res], np.int64)}


def _train_data(c, seed):
    """Training pairs as mlp_features makes them of converged weights, and the
    parameters of a fresh network (uniform in +-1/sqrt(fan in))."""
    rng = np.random.default_rng(seed)
    xs, ts, left = [], [], c["points"]
    while left > 0:
        L = 8 * int(rng.integers(2, 17))
        x, t = m.mlp_features(L, rng.uniform(0.4, 0.8), rng.uniform(1.9, 2.0), _weights(L, int(rng.integers(1 << 30))))
        xs.append(x[:left])
        ts.append(t[:left])
        left -= len(xs[-1])
    p = [rng.uniform(-1.0, 1.0, n) / math.sqrt(fan) for fan, n in
         ((4, 4 * 128 + 128), (128, 128 * 129), (128, 128 * 129), (128, 129))]
    return np.concatenate(xs), np.concatenate(ts), np.concatenate(p).astype(np.float32)


def _prepare_train(c, seed):
    x, t, p = _train_data(c, seed)
    net = m.MLP()
    net.set_params(p)
    net.set_data(x, t)
    return {"net": net, "p": p, "c": c, "seed": seed & 0xFFFF}


def _run_train(s):
    net, c = s["net"], s["c"]
    net.set_params(s["p"])
    losses = net.train(c["steps"], batch=c["batch"], lr=c["lr"], seed=s["seed"])
    return {"losses": losses, "params": net.params()}


def _hist2d(L, seed):
    """Counts of a production run: every row (E_Delta) visited about equally,
    spread over its magnetisations, with some rows empty."""
    N = L * L
    n = (N + 1) * (N + 2) // 2
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    h = torch.randint(0, 4000, (n,), generator=g, device="cuda", dtype=torch.int64)
    h.mul_(torch.randint(0, 4, (n,), generator=g, device="cuda", dtype=torch.int64).eq_(0))
    row = N // 3
    h[row * (row + 1) // 2:(row + 1) * (row + 2) // 2] = 0
    return h


def _deltas(c):
    return [1.95 + 0.01 * k for k in range(c["deltas"])]


def _shifted(c, seed):
    """The weights shifted for each Delta point, as weight_shift does: the
    largest Boltzmann factor of the rows becomes 1."""
    w = _weights(c["L"], seed)
    i = np.arange(w.size)
    return np.stack([w + (-w - BETA * d * i).max() for d in _deltas(c)])


def _prepare_reweight(c, seed):
    return {"L": c["L"], "hist": _hist2d(c["L"], seed), "lnw": torch.from_numpy(_shifted(c, seed)).cuda(),
            "sums": torch.zeros(c["deltas"], 4, dtype=torch.float64, device="cuda"), "deltas": _deltas(c)}


def _run_reweight(s):
    stream = torch.cuda.current_stream().cuda_stream
    for k, d in enumerate(s["deltas"]):
        m.observables_noalloc(0, s["hist"].data_ptr(), s["lnw"][k].data_ptr(), s["L"], BETA, d,
                              s["sums"][k].data_ptr(), stream)
    return s["sums"]


_PREPARE = {"iterate": _prepare_iterate, "run": _prepare_run, "produce": _prepare_produce, "random": _prepare_random,
            "batch": _prepare_batch, "train": _prepare_train, "reweight": _prepare_reweight}
_RUN = {"iterate": _run_iterate, "run": _run_run, "produce": _run_produce, "random": _run_random, "batch": _run_batch,
        "train": _run_train, "reweight": _run_reweight}


def prepare(case, seed):
    s = _PREPARE[case["kind"]](case, seed)
    s["run"] = _RUN[case["kind"]]
    return s


def run(state):
    return state["run"](state)


# ---- what a pass cannot do without ----------------------------------------

# integer and FP32 operations of one Metropolis attempt: half a Philox4x32-7
# block (7 rounds of 2 multiplications and 4 exclusive-ors), the proposal, the
# neighbour sum, the logarithm, the comparison and the running sums
ATTEMPT_OPS = 41


def work(case):
    k = case["kind"]
    if k == "train":
        P, n = 33793, case["batch"] * case["steps"]
        return {"bytes": n * 20 + case["steps"] * P * 4 * 6, "flops": n * 6 * 33664}
    L = case.get("L", 0)
    N = L * L
    if k == "reweight":
        bins = (N + 1) * (N + 2) // 2
        return {"bytes": case["deltas"] * (bins + N + 1) * 8, "flops": case["deltas"] * bins * 8}
    if k == "batch":
        sizes = list(range(case["Lmin"], case["Lmax"] + 1, 8))
        Ns = [sizes[i % len(sizes)] ** 2 for i in range(case["instances"])]
        att = sum(2 * x * case["chains"] * case["iters"] for x in Ns)
        return {"bytes": sum(case["chains"] * x // 2 + (x + 1) * 24 for x in Ns), "flops": att * ATTEMPT_OPS}
    c = case["chains"]
    lattice = c * N // 2 + c * 24  # 2 bits per spin in and out, E_J, E_Delta, M in and out
    if k == "run":
        att = c * case["iters"] * (N + case["starting_M"])
        return {"bytes": lattice + (N + 1) * 24, "flops": att * ATTEMPT_OPS}
    if k == "produce":
        return {"bytes": lattice + (N + 1) * (N + 2) // 2 * 16 + (N + 1) * 8, "flops": c * 2 * N * ATTEMPT_OPS}
    return {"bytes": lattice + (N + 1) * 24, "flops": c * (N if k == "random" else 2 * N) * ATTEMPT_OPS}


# ---- the same in 64 bits ----------------------------------------------------

def _philox4x32_10(ctr0, ctr1, ctr2, ctr3, key0, key1):
    """Word 0 of Philox4x32-10 (Salmon et al., SC'11) for an array of ctr0."""
    M0, M1, mask = np.uint64(0xD2511F53), np.uint64(0xCD9E8D57), np.uint64(0xFFFFFFFF)
    x = [np.asarray(ctr0, np.uint64)] + [np.full(len(ctr0), v, np.uint64) for v in (ctr1, ctr2, ctr3)]
    for r in range(10):
        k0, k1 = np.uint64((key0 + r * 0x9E3779B9) & 0xFFFFFFFF), np.uint64((key1 + r * 0xBB67AE85) & 0xFFFFFFFF)
        p0, p1 = M0 * x[0], M1 * x[2]
        x = [(p1 >> np.uint64(32)) ^ x[1] ^ k0, p1 & mask, (p0 >> np.uint64(32)) ^ x[3] ^ k1, p0 & mask]
    return x[0]


def _exact_train(c, seed):
    x, t, p = _train_data(c, seed)
    X, T = torch.from_numpy(x).cuda().double(), torch.from_numpy(t).cuda().double()
    P = torch.from_numpy(p).cuda().double().requires_grad_(True)
    mom, var = torch.zeros_like(P), torch.zeros_like(P)
    b1, b2, eps = 0.9, 0.999, 1e-8
    losses = []
    for step in range(c["steps"]):
        r = _philox4x32_10(np.arange(c["batch"]), step, 0x57A27, 0, seed & 0xFFFF, 0x4D4C5000)
        idx = torch.from_numpy(((r * np.uint64(len(x))) >> np.uint64(32)).astype(np.int64)).cuda()
        h, off = X[idx], 0
        for layer, (o, i) in enumerate(((128, 4), (128, 128), (128, 128), (1, 128))):
            z = h @ P[off:off + o * i].view(o, i).T + P[off + o * i:off + o * i + o]
            h = torch.nn.functional.silu(z) if layer < 3 else z
            off += o * i + o
        loss = ((h[:, 0] - T[idx]) ** 2).mean()
        (g,) = torch.autograd.grad(loss, P)
        losses.append(float(loss.detach()))
        with torch.no_grad():
            mom = b1 * mom + (1 - b1) * g
            var = b2 * var + (1 - b2) * g * g
            P -= c["lr"] * (mom / (1 - b1 ** (step + 1))) / ((var / (1 - b2 ** (step + 1))).sqrt() + eps)
    return {"losses": np.array(losses), "params": P.detach().cpu().numpy()}


def _exact_reweight(c, seed):
    L = c["L"]
    N = L * L
    h, lnw = _hist2d(L, seed), _shifted(c, seed)
    rows = torch.zeros(4, N + 1, dtype=torch.float64, device="cuda")
    a = torch.arange(-N, N + 1, device="cuda", dtype=torch.float64).abs_()
    for i in range(N + 1):
        r = h[i * (i + 1) // 2:(i + 1) * (i + 2) // 2].double()
        am = a[N - i:N + i + 1:2]
        m2 = am * am
        rows[0, i], rows[1, i], rows[2, i], rows[3, i] = r.sum(), (r * am).sum(), (r * m2).sum(), (r * m2 * m2).sum()
    rows = rows.cpu().numpy()
    i = np.arange(N + 1, dtype=np.float64)
    return np.stack([(rows * np.exp(-BETA * d * i - lnw[k])).sum(axis=1) for k, d in enumerate(_deltas(c))])


def exact(case, seed):
    """The training steps and the reweighting sums.  The other kinds return
    counts and integer state of a random walk, and weights that follow from
    those counts: they have no value apart from the walk itself."""
    if case["kind"] == "train":
        return _exact_train(case, seed)
    if case["kind"] == "reweight":
        return _exact_reweight(case, seed)
    return None
