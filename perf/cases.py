"""The performance cases: the work a search over this library has it do.

Each case is one call of the public evaluator API (`GpuEvaluator`,
`GenomePool`) on a resident dataset, with the programs and fit plans that a
search holds when it makes the call. The families:

  screen    the fixed-width pool of a generation, scored (GenomePool.score);
  score     a packed batch of programs scored under one objective;
  fit       batched constant fitting (LM, L1 / log-squashed IRLS, correlation);
  impscore  the implicit metric |f| / |grad f| of a batch;
  impfit    its constant fitting;
  rank      exact rank-correlation sums of a batch;
  median    the exact median of |residual| of a batch;
  vary      the next generation of the pool.

Sizes are those of the repository's own configurations and tests, from the
plain-method search (4 islands x 200 programs over 8,000 training rows) to the
batches over a million rows and more; data and programs come from
`workloads.py`, seeded.
"""
import importlib
import math

import numpy as np
import torch

pkg = importlib.import_module("the-rule-and-compass_b200")
W = importlib.import_module("the-rule-and-compass_b200.workloads")
E = pkg.expr

# objective and metric codes of the evaluator
SCORE_KINDS = {"squared": 0, "absolute": 1, "log_squashed": 2, "maximum": 4, "correlation": 5,
               "log_loss": 10}
FIT_METRICS = {"squared": 0, "log_squashed": 1, "correlation": 2, "absolute": 4}

# mean postfix ops per program of the generators, for work()
OPS = {"screen": 12, "score": 12, "fit": 33, "impscore": 22, "impfit": 24, "rank": 33,
       "median": 33}


def listed():
    return [
        # One generation's screen in the plain-method search: 4 islands x 200
        # random programs, one input, the 80 % training split of 10,000 rows.
        # Latency, launches and the longest program decide.
        {"name": "screen_small", "family": "screen", "islands": 4, "pop": 200, "rows": 8000,
         "inputs": 1, "objective": "squared"},
        # A handful of classification candidates with row weights, over an odd
        # number of rows: the smallest scoring calls.
        {"name": "score_labels_few", "family": "score", "programs": 24, "rows": 20011,
         "inputs": 5, "objective": "log_loss"},
        # The headline scoring batch.
        {"name": "score_batch", "family": "score", "programs": 4096, "rows": 1048576,
         "inputs": 5, "objective": "squared"},
        # An ordinary screen under a two-pass objective, ragged sizes.
        {"name": "score_corr", "family": "score", "programs": 701, "rows": 131101, "inputs": 8,
         "objective": "correlation"},
        # The admitted candidates of one generation of the plain-method search,
        # 8 LM iterations: a short fit that waits on its own steps.
        {"name": "fit_small", "family": "fit", "programs": 56, "rows": 8000, "inputs": 1,
         "metric": "squared", "iters": 8, "source": "pool"},
        # The fused fit of 1-20 constants over 8 inputs.
        {"name": "fit_batch", "family": "fit", "programs": 512, "rows": 262144, "inputs": 8,
         "metric": "squared", "iters": 20, "source": "trees"},
        # L1 IRLS over heavy-tailed inputs.
        {"name": "fit_l1", "family": "fit", "programs": 96, "rows": 1048576, "inputs": 10,
         "metric": "absolute", "iters": 20, "source": "trees"},
        # The implicit metric on a noisy circle: value and input gradient.
        {"name": "implicit_score", "family": "impscore", "programs": 256, "rows": 1048576},
        # Its constant fit (second-order reverse sweeps in f64).
        {"name": "implicit_fit", "family": "impfit", "programs": 48, "rows": 131072,
         "iters": 20},
        # Rank correlation of fitted candidates, the heavy-tailed inputs.
        {"name": "rank_batch", "family": "rank", "programs": 32, "rows": 2097152},
        # The median-error metric: ordinary sizes, odd row count.
        {"name": "median_batch", "family": "median", "programs": 33, "rows": 300007},
        # One generation of the pool at the size of the heavy-tailed search.
        {"name": "vary", "family": "vary", "islands": 16, "pop": 1000, "inputs": 10},
    ]


def _log(rng, lo, hi):
    """An integer spread over the logarithm of [lo, hi]."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    f = rng.choice(["screen", "score", "score", "fit", "fit", "impscore", "impfit", "rank",
                    "median", "vary"])
    if f == "screen":
        return {"family": f, "islands": rng.randint(1, 16), "pop": _log(rng, 24, 1000),
                "rows": _log(rng, 1000, 262144), "inputs": rng.randint(1, 10),
                "objective": rng.choice(["squared", "absolute"])}
    if f == "score":
        return {"family": f, "programs": _log(rng, 8, 4096), "rows": _log(rng, 4000, 1048576),
                "inputs": rng.randint(3, 10), "objective": rng.choice(sorted(SCORE_KINDS))}
    if f == "fit":
        rows = _log(rng, 4000, 1048576)
        most = min(512, max(16, (1 << 26) // rows))
        return {"family": f, "programs": _log(rng, 8, most), "rows": rows,
                "inputs": rng.randint(3, 10), "metric": rng.choice(sorted(FIT_METRICS)),
                "iters": rng.choice([8, 20]), "source": rng.choice(["pool", "trees"])}
    if f == "impscore":
        # whole 64-row groups: what one warp of the implicit scorer takes a step
        return {"family": f, "programs": _log(rng, 16, 512),
                "rows": 64 * _log(rng, 64, 16384)}
    if f == "impfit":
        rows = _log(rng, 4000, 131072)
        return {"family": f, "programs": _log(rng, 8, min(96, max(9, (3 << 21) // rows))),
                "rows": rows, "iters": rng.choice([8, 20])}
    if f == "rank":
        rows = _log(rng, 4000, 2097152)
        return {"family": f, "programs": _log(rng, 4, min(400, max(5, (1 << 26) // rows))),
                "rows": rows}
    if f == "median":
        rows = _log(rng, 4000, 1048576)
        return {"family": f, "programs": _log(rng, 4, min(200, max(5, (1 << 25) // rows))),
                "rows": rows}
    return {"family": f, "islands": rng.randint(1, 16), "pop": _log(rng, 50, 1000),
            "inputs": rng.randint(1, 10)}


# ---- inputs ---------------------------------------------------------------

def _data(case, seed):
    """(x f64 [v][n], y f64 [n]) of the case."""
    f, n = case["family"], case["rows"]
    if f in ("impscore", "impfit"):
        return W.implicit_data(n, seed), np.zeros(n)
    if f in ("rank", "median") or case.get("metric") == "absolute":
        x, y = W.heavy_tail_data(n, seed)
        return x[: case.get("inputs", 10)], y
    if f == "fit" and case["inputs"] > 1:
        return W.fit_data(n, seed, case["inputs"])
    if case["inputs"] == 1:  # the plain-method search's line
        rng = np.random.Generator(np.random.PCG64(seed))
        x = rng.uniform(-5.0, 5.0, n)
        return x[None, :], 2.0 * x + 1.0 + rng.normal(0.0, 0.1, n)
    rng = np.random.Generator(np.random.PCG64(seed))
    x = rng.standard_normal((case["inputs"], n)).astype(np.float32).astype(np.float64)
    v = case["inputs"]
    y = x[0] * x[1 % v] + np.sin(x[2 % v]) + rng.normal(0.0, 0.05, n)
    if case.get("objective") == "log_loss":
        y = (y > 0.0).astype(np.float64)
    return x, y.astype(np.float32).astype(np.float64)


def _labels(case, y, seed):
    """Label signs and row weights (some zero) of a classification case."""
    rng = np.random.Generator(np.random.PCG64(seed + 77))
    w = rng.uniform(0.0, 2.0, len(y))
    w[rng.random(len(y)) < 0.1] = 0.0
    return 2.0 * y - 1.0, w


def _trees(case, seed):
    f, p = case["family"], case["programs"]
    if f == "score":
        rng = np.random.Generator(np.random.PCG64(seed + 1000))
        return [W.random_scoring_tree(rng, case["inputs"]) for _ in range(p)]
    if f == "impscore":
        return W.implicit_workload(p, 1, seed)[0]
    return W.fit_workload(p, 1, seed, nvars=case.get("inputs", 10))[0]


def _evaluator(x, y):
    ev = pkg.GpuEvaluator(x.astype(np.float32).reshape(-1), x.shape[1], x.shape[0],
                          y.astype(np.float32))
    return ev


def _random_pool(ev, islands, pop, inputs, seed):
    """A pool whose buffer 1 holds a restarted (random) population, and its
    words."""
    width = pkg.width_for(30)
    n = islands * pop
    pool = pkg.GenomePool(ev, islands, pop, width)
    words = np.full((n, width), E.HALT, np.uint32)
    words[:, 0], words[:, 1] = E.VAR, 0
    pool.upload(0, words)
    out = pool.vary(0, np.zeros(n), 0, inputs, 30, seed & 0x7fffffff,
                    pkg.DEFAULT_VARIATION_OPS, restart=[1] * islands)
    return pool, out[0]


def prepare(case, seed):
    f = case["family"]
    if f == "vary":
        x = np.linspace(-1.0, 1.0, 64, dtype=np.float32)
        ev = pkg.GpuEvaluator(np.stack([x] * case["inputs"]).reshape(-1), 64, case["inputs"], x)
        pool, _ = _random_pool(ev, case["islands"], case["pop"], case["inputs"], seed)
        n = case["islands"] * case["pop"]
        err = np.random.Generator(np.random.PCG64(seed)).random(n)
        return {"case": case, "ev": ev, "pool": pool, "err": err, "seed": seed & 0x7fffffff}
    x, y = _data(case, seed)
    ev = _evaluator(x, y)
    s = {"case": case, "ev": ev}
    if f == "screen":
        s["pool"], s["words"] = _random_pool(ev, case["islands"], case["pop"], case["inputs"],
                                             seed)
        return s
    if f == "score":
        if case["objective"] == "log_loss":
            sign, w = _labels(case, y, seed)
            ev.set_fit_sign(sign)
            ev.set_score_weights(w)
        s["prog"], s["off"] = pkg.Population(_trees(case, seed)).programs()
        return s
    ev.set_fit_data(x.reshape(-1), y)
    if f == "fit" and case["source"] == "pool":
        p = case["programs"]
        # (about half of the random programs hold constants)
        _, words = _random_pool(ev, 16, max(8, p // 4), case["inputs"], seed)
        plans = [q for q in pkg.host.gpu_fit_plans_words(words) if not isinstance(q, str)]
        s["plans"] = plans[:p]
    elif f == "fit":
        s["plans"] = [pkg.gpu_fit_plan(t) for t in _trees(case, seed)]
    elif f == "impfit":
        trees = W.implicit_workload(2 * case["programs"] + 8, 1, seed)[0]
        trees = [t for t in trees if t.constants()][: case["programs"]]
        s["plans"] = [pkg.gpu_fit_plan(t) for t in trees]
    else:
        plans = [pkg.gpu_fit_plan(t, allow_no_constants=True) for t in _trees(case, seed)]
        s["packed"] = pkg.pack_plans(plans)
    return s


# ---- the calls ------------------------------------------------------------

def run(s):
    case, ev = s["case"], s["ev"]
    f = case["family"]
    if f == "screen":
        value, status, _ = s["pool"].score(1, SCORE_KINDS[case["objective"]])
        return {"value": value, "status": status}
    if f == "score":
        value, status, _ = ev.score_batch(s["prog"], s["off"], SCORE_KINDS[case["objective"]])
        return {"value": value, "status": status}
    if f in ("fit", "impfit"):
        metric = FIT_METRICS[case["metric"]] if f == "fit" else 6
        c, loss, status, _ = ev.fit_plans(s["plans"], case["iters"], metric)
        constants = np.zeros((len(loss), 20))  # the columns are the batch's own maximum
        constants[:, : c.shape[1]] = c
        return {"constants": constants, "loss": loss, "status": status}
    if f == "vary":
        words, length, cost, hashes, err, _ = s["pool"].vary(
            1, s["err"], 1, case["inputs"], 30, s["seed"], pkg.DEFAULT_VARIATION_OPS)
        return {"words": words.view(np.int32), "length": length.view(np.int16),
                "cost": cost.view(np.int16), "hash": hashes.view(np.int64), "error": err}
    prog, off, pcount, c0, _, kmax = s["packed"]
    if f == "impscore":
        value, status, _ = ev.implicit_score(prog, off, pcount, c0, kmax)
        return {"value": value, "status": status}
    if f == "median":
        value, status, _ = ev.order_stat(prog, off, pcount, c0, kmax, 0)
        return {"value": value, "status": status}
    sums, status, bb, _ = ev.rank_sums(prog, off, pcount, c0, kmax)
    # the sums are up to 2^65: each as two whole numbers
    parts = [(v >> 32, v & 0xffffffff) for ab, aa in (t or (0, 0) for t in sums)
             for v in (ab, aa)] + [(bb >> 32, bb & 0xffffffff)]
    return {"sums": np.asarray(parts, np.int64), "status": status}


def work(case):
    """Bytes: rows and programs in, results out; flops: one lane operation
    per postfix op and row (an adjoint 2.5 more), for fits times the
    iterations, with the Gram products of about ten constants."""
    f = case["family"]
    if f == "vary":
        n = case["islands"] * case["pop"]
        return {"bytes": n * (2 * 64 * 4 + 28.0), "flops": n * 300.0}
    n = case["rows"]
    p = case["programs"] if "programs" in case else case["islands"] * case["pop"]
    ops = OPS[f]
    v = case.get("inputs", 4 if f.startswith("imp") else 10)
    width = 4.0 if f in ("screen", "score", "impscore") else 12.0
    io = n * (v + 1) * width + p * (8.0 * ops + 12.0)
    if f in ("screen", "score"):
        return {"bytes": io, "flops": float(p) * n * (ops + 2)}
    if f == "impscore":
        return {"bytes": io, "flops": float(p) * n * (3.5 * ops + 6)}
    if f in ("fit", "impfit"):
        gram = 2 * (10 * 11 / 2 + 11)
        return {"bytes": io, "flops": float(p) * n * case["iters"] * (4.5 * ops + gram)}
    return {"bytes": io + (16.0 * p * n if f == "rank" else 0.0), "flops": float(p) * n * (ops + 8)}


# ---- the same results in 64 bits ------------------------------------------

def _postfix_of_tree(t, f32):
    out = []

    def walk(q):
        for k in q.kids:
            walk(k)
        out.append((q.op, float(np.float32(q.val)) if f32 and q.op == E.CONST else q.val))
    walk(t)
    return out


def _postfix_of_words(words):
    out, i = [], 0
    while words[i] != E.HALT:
        op = int(words[i])
        if op in (E.CONST, E.VAR):
            a = words[i + 1]
            out.append((op, float(a.view(np.float32)) if op == E.CONST else int(a)))
            i += 2
        else:
            out.append((op, 0.0))
            i += 1
    return out


def _evaluate(prog, cols):
    """One postfix program over all rows in f64, with the guards of the
    expression semantics (an undefined value is not a number)."""
    nan = torch.full((), float("nan"), dtype=torch.float64, device=cols[0].device)
    st = []
    for op, val in prog:
        if op == E.CONST:
            st.append(torch.full_like(cols[0], val))
        elif op == E.VAR:
            st.append(cols[int(val)])
        elif op == E.IF:
            b, a, c = st.pop(), st.pop(), st.pop()
            st.append(torch.where(c > 0, a, b))
        elif op in E.BINARY:
            b, a = st.pop(), st.pop()
            if op == E.ADD:
                r = a + b
            elif op == E.SUB:
                r = a - b
            elif op == E.MUL:
                r = a * b
            elif op == E.DIV:
                r = torch.where(b.abs() < 1e-12, nan, a / b)
            elif op == E.POW:
                r = torch.where((a < 0) & ((b - b.round()).abs() > 1e-9), nan, torch.pow(a, b))
            else:
                raise ValueError(op)
            st.append(r)
        else:
            a = st.pop()
            if op == E.LOG:
                r = torch.where(a > 0, a.log(), nan)
            elif op == E.EXP:
                r = torch.where(a > 700, math.inf, a.exp())
            else:
                r = {E.SIN: torch.sin, E.COS: torch.cos, E.TAN: torch.tan, E.SQRT: torch.sqrt,
                     E.ABS: torch.abs, E.TANH: torch.tanh, E.SIG: torch.sigmoid,
                     E.SQUARE: lambda q: q * q, E.CUBE: lambda q: q * q * q, E.NEG: torch.neg,
                     E.GAUSS: lambda q: (-q * q).exp(), E.SINH: torch.sinh,
                     E.COSH: torch.cosh}[op](a)
            st.append(r)
    return st.pop()


def _score(p, y, objective, sign, w):
    if objective == "log_loss":
        use = w > 0
        p, sign, w = p[use], sign[use], w[use]
    if not bool(torch.isfinite(p).all()) or float(p.abs().max()) > 1e30:
        return math.inf
    r = p - y if objective != "log_loss" else None
    if objective == "squared":
        return float((r * r).mean())
    if objective == "absolute":
        return float(r.abs().mean())
    if objective == "log_squashed":
        return float(torch.log1p(r * r).mean())
    if objective == "maximum":
        return float(r.abs().max())
    if objective == "log_loss":
        u = sign * p
        return float((w * (torch.relu(-u) + torch.log1p(torch.exp(-u.abs())))).sum() / w.sum())
    dp, dy = p - p.mean(), y - y.mean()
    sp, sy = float((dp * dp).sum()), float((dy * dy).sum())
    if sp <= 0 or sy <= 0:
        return 1.0
    return 1.0 - abs(float((dp * dy).sum())) / (math.sqrt(sp) * math.sqrt(sy))


def exact(case, seed):
    """Scores, implicit scores and medians from plain f64 torch; the fits
    (trajectories of an iteration), the rank sums and the variation (whole
    numbers) have no such value."""
    f = case["family"]
    if f in ("fit", "impfit", "rank", "vary"):
        return None
    gpu = torch.cuda.is_available()
    p = case["programs"] if "programs" in case else case["islands"] * case["pop"]
    if not gpu and p * case["rows"] > 1e8:
        return None
    dev = "cuda" if gpu else "cpu"
    x, y = _data(case, seed)
    if f == "median":
        cols = [torch.from_numpy(np.ascontiguousarray(c)).to(dev) for c in x]
        yt = torch.from_numpy(y).to(dev)
    else:
        cols = [torch.from_numpy(c.astype(np.float32).astype(np.float64)).to(dev) for c in x]
        yt = torch.from_numpy(y.astype(np.float32).astype(np.float64)).to(dev)
    if f == "screen":
        progs = [_postfix_of_words(q) for q in prepare(case, seed)["words"]]
    else:
        progs = [_postfix_of_tree(t, f == "score") for t in _trees(case, seed)]
    value = np.zeros(len(progs))
    sign = w = None
    if case.get("objective") == "log_loss":
        sign, w = (torch.from_numpy(a).to(dev) for a in _labels(case, y, seed))
    for k, prog in enumerate(progs):
        if f in ("screen", "score"):
            value[k] = _score(_evaluate(prog, cols), yt, case["objective"], sign, w)
        elif f == "median":
            r = (_evaluate(prog, cols) - yt).abs()
            if not bool(torch.isfinite(r).all()):
                value[k] = math.nan
                continue
            r = r.sort().values
            n = len(r)
            value[k] = float(r[n // 2]) if n % 2 else 0.5 * float(r[n // 2 - 1] + r[n // 2])
        else:
            leaves = [c.clone().requires_grad_(True) for c in cols]
            v = _evaluate(prog, leaves)
            if v.requires_grad:
                g = torch.autograd.grad(v.sum(), leaves, allow_unused=True)
                norm = sum(q * q for q in g if q is not None).sqrt()
            else:
                norm = torch.zeros_like(cols[0])
            d = v.detach().abs() / norm
            ok = bool((torch.isfinite(d) & (norm > 0) & torch.isfinite(norm)).all())
            value[k] = float(d.mean()) if ok else math.inf
    return {"value": value, "status": None}
