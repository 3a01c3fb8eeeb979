"""The work that users of this solver have it do, as measurable cases.

Every case goes through the package's public entry points (`lnorm`,
`solve_reduced`, `Batch`, `learned.solve_learned_batch`, `Mlp`).  Sizes and
value distributions are those of the repository's five benchmark
configurations (`workloads.py`), its tests and its wide-matrix workload, from
solves that end before a launch is noticed to ones of tens of milliseconds.

kinds
    text      matrix text in, value and strategy out (what the `L_CUDA`
              executable does: parse, preprocess, solve, report)
    solve     one exhaustive solve of a matrix in memory
    batch     many matrices of uneven size in one kept `Batch`
    learned   exact solves of 44-column low-rank matrices that start from
              the proposal network's labelings
    gradient  forward and backward pass of the proposal network

value distributions
    uniform   integers in [-amp, amp]
    pm1       entries -1 and +1
    sparse    entries -1, 0, 1 with a marginal row and column in [-5, 5]
    gauss     round(N(0, amp^2))
    lowrank   round(5 U V) + integers in [-2, 2], rank 3
"""
import importlib
import math

import numpy as np

PKG = "l-norms_bruteforce_b200"


def _ld():
    return importlib.import_module(PKG)


def _learned():
    return importlib.import_module(PKG + ".learned")


def listed():
    return [
        # the smallest call: a witness of a few settings, where the launch and the host path are the time
        {"name": "solve_l1_14x16", "kind": "solve", "rows": 14, "cols": 16, "d": 1, "marginal": False,
         "values": "uniform", "amp": 10},
        # configuration 1: the everyday small Bell matrix, from its text file's content to the strategy
        {"name": "text_l1_24x24", "kind": "text", "rows": 24, "cols": 24, "d": 1, "marginal": False,
         "values": "uniform", "amp": 10, "flag": "n", "copies": 0},
        # configuration 2: Bell expression with marginals, duplicated and zero lines, uniting on
        {"name": "text_lm_34x37", "kind": "text", "rows": 34, "cols": 37, "d": 1, "marginal": True,
         "values": "sparse", "amp": 1, "flag": "y", "copies": 4},
        # correlation-type Bell matrix of +-1 entries, an odd size
        {"name": "solve_l1_35x33_pm1", "kind": "solve", "rows": 35, "cols": 33, "d": 1, "marginal": False,
         "values": "pm1", "amp": 1},
        # the plain enumeration of configuration 5's distribution, at a size solved in one sitting; the largest case
        {"name": "solve_l1_35x44_lowrank", "kind": "solve", "rows": 35, "cols": 44, "d": 1, "marginal": False,
         "values": "lowrank", "amp": 5},
        # two-message prepare-and-measure witness with large coefficients, ragged width
        {"name": "solve_l2_30x43_gauss", "kind": "solve", "rows": 30, "cols": 43, "d": 2, "marginal": False,
         "values": "gauss", "amp": 20},
        # configuration 3: three messages, +-1 entries
        {"name": "solve_l3_20x30_pm1", "kind": "solve", "rows": 20, "cols": 30, "d": 3, "marginal": False,
         "values": "pm1", "amp": 1},
        # more messages than the configurations use: a short solve
        {"name": "solve_l4_14x20", "kind": "solve", "rows": 14, "cols": 20, "d": 4, "marginal": False,
         "values": "uniform", "amp": 3},
        # more columns than one thread holds (the wide-matrix workload)
        {"name": "solve_l1_28x200_wide", "kind": "solve", "rows": 28, "cols": 200, "d": 1, "marginal": False,
         "values": "uniform", "amp": 40},
        # configuration 4: a batch of matrices of uneven n, m and d in one launch
        {"name": "batch_256", "kind": "batch", "count": 256, "max_rows": 24},
        # configuration 5: exact 44 x 44 solves from learned incumbents
        {"name": "learned_44x44", "kind": "learned", "count": 8, "rows": 44, "directions": 8},
        # one training batch of the proposal network: loss and every gradient
        {"name": "gradient_1024", "kind": "gradient", "rows": 1024},
    ]


def _log_int(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


# no drawn case does more than the largest listed one
_MOST = 2.0 * 44 * 2.0 ** 34


def draw(rng):
    """One more case: the kinds, options and sizes of the listed ones, spread over their ranges."""
    while True:
        kind = rng.choice(["text", "solve", "solve", "solve", "solve", "wide", "batch", "learned", "gradient"])
        if kind == "batch":
            case = {"kind": "batch", "count": _log_int(rng, 24, 256), "max_rows": rng.randint(18, 24)}
        elif kind == "learned":
            case = {"kind": "learned", "count": rng.randint(1, 8), "rows": rng.randint(36, 44),
                    "directions": rng.choice([2, 4, 8, 16])}
        elif kind == "gradient":
            case = {"kind": "gradient", "rows": _log_int(rng, 100, 1024)}
        elif kind == "wide":
            case = {"kind": "solve", "rows": rng.randint(18, 29), "cols": rng.randint(65, 256), "d": rng.choice([1, 1, 2]),
                    "marginal": False, "values": "uniform", "amp": rng.randint(1, 40)}
        elif kind == "text":
            marginal = rng.random() < 0.5
            case = {"kind": "text", "rows": rng.randint(16, 34), "cols": rng.randint(36, 44), "d": 1,
                    "marginal": marginal, "values": "sparse" if marginal else "uniform",
                    "amp": 1 if marginal else rng.randint(1, 10), "flag": rng.choice("ny"),
                    "copies": rng.randint(0, 4)}
        else:
            d = rng.choice([1, 1, 1, 2, 2, 3, 3, 4, 5])
            rows = {1: (12, 35), 2: (12, 32), 3: (8, 20), 4: (6, 14), 5: (6, 12)}[d]
            cols = (12, 64) if d < 4 else (8, 30)
            values = rng.choice(["uniform", "uniform", "pm1", "gauss"] + (["lowrank"] if d == 1 else []))
            case = {"kind": "solve", "rows": rng.randint(*rows), "cols": rng.randint(*cols), "d": d, "marginal": False,
                    "values": values,
                    "amp": {"uniform": _log_int(rng, 1, 40), "pm1": 1, "gauss": rng.randint(5, 20), "lowrank": 5}[values]}
        if work(case)["flops"] <= _MOST:
            return case


# ---- inputs ------------------------------------------------------------------

def _entries(rng, rows, cols, values, amp):
    if values == "uniform":
        return rng.integers(-amp, amp + 1, size=(rows, cols), dtype=np.int64)
    if values == "pm1":
        return rng.choice(np.array([-1, 1], dtype=np.int64), size=(rows, cols))
    if values == "gauss":
        return np.rint(rng.normal(0.0, amp, size=(rows, cols))).astype(np.int64)
    if values == "lowrank":
        u, v = rng.standard_normal((rows, 3)), rng.standard_normal((3, cols))
        return np.rint(amp * (u @ v)).astype(np.int64) + rng.integers(-2, 3, size=(rows, cols), dtype=np.int64)
    a = rng.integers(-1, 2, size=(rows, cols), dtype=np.int64)          # sparse
    a[0, :] = rng.integers(-5, 6, size=cols)
    a[:, 0] = rng.integers(-5, 6, size=rows)
    return a


def _matrix(case, rng):
    a = _entries(rng, case["rows"], case["cols"], case["values"], case["amp"])
    for _ in range(case.get("copies", 0)):     # repeated and zero rows, as the uniting flag is used for
        i, j = int(rng.integers(1, a.shape[0])), int(rng.integers(1, a.shape[0] + 1))
        a = np.insert(a, j, a[i] if rng.random() < 0.7 else np.zeros(a.shape[1], np.int64), axis=0)
    if case.get("copies", 0) and case.get("flag") != "y":
        a = a[:case["rows"]]                   # without uniting, repeated rows cost labelings
    return a


def _batch_inputs(case, rng):
    mats, ds = [], []
    for _ in range(case["count"]):
        d = int(rng.choice(np.array([1, 2, 3]), p=np.array([0.6, 0.3, 0.1])))
        n = int(rng.integers(16, (case["max_rows"] if d < 3 else 17) + 1))
        m = int(rng.integers(16, 65))
        mats.append(np.rint(rng.normal(0.0, 20.0, size=(n, m))).astype(np.int64))
        ds.append(d)
    return mats, ds


def _net_inputs(case, seed):
    rng = np.random.default_rng(seed)
    rows, width = case["rows"], 44
    x = rng.standard_normal((rows, 3)) @ rng.standard_normal((3, width))
    x = x / np.sqrt(np.mean(x * x, axis=1, keepdims=True))
    mask = np.zeros((rows, width), np.float32)
    for r, n in enumerate(rng.integers(16, 29, size=rows)):
        mask[r, rng.permutation(width)[:n]] = 1.0
    x = (np.clip(x, -8.0, 8.0) * mask).astype(np.float32)
    t = ((x + 0.3 * rng.standard_normal((rows, width))) > 0).astype(np.float32) * mask
    params = {}
    for name, (o, i) in {"1": (256, 44), "2": (256, 256), "3": (44, 256)}.items():
        lim = math.sqrt(6.0 / i)
        params["W" + name] = rng.uniform(-lim, lim, (o, i)).astype(np.float32)
        params["b" + name] = rng.normal(0.0, 0.05, o).astype(np.float32)
    return params, x, t, mask


SKIP = 4.0   # weight of the network's residual path, as learned.py trains it


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    ld = _ld()
    kind = case["kind"]
    if kind == "text":
        a = _matrix(case, rng)
        return {"case": case, "text": "".join(" ".join(str(int(v)) for v in row) + "\n" for row in a)}
    if kind == "solve":
        return {"case": case, "a": _matrix(case, rng)}
    if kind == "batch":
        mats, ds = _batch_inputs(case, rng)
        return {"case": case, "batch": ld.Batch(mats, ds)}
    if kind == "learned":
        mats = [_entries(rng, case["rows"], 44, "lowrank", 5) for _ in range(case["count"])]
        return {"case": case, "mats": mats,
                "proposer": _learned().Proposer("network", directions=case["directions"])}
    params, x, t, mask = _net_inputs(case, seed)
    net = ld.Mlp(batch=-(-case["rows"] // 128) * 128, seed=0, skip=SKIP)
    net.set_params(params)
    return {"case": case, "net": net, "x": x, "t": t, "mask": mask}


def _solution(s):
    return {"value": np.int64(s.value), "gray_index": np.uint64(s.gray_index), "labels": np.asarray(s.labels)}


def run(state):
    case = state["case"]
    ld = _ld()
    kind = case["kind"]
    if kind == "text":
        value, _, _, strategy = ld.lnorm(state["text"], case["d"], case["flag"], case["marginal"])
        return {"value": np.int64(value), "strategy": np.array(strategy.split(), dtype=np.int64)}
    if kind == "solve":
        return _solution(ld.solve_reduced(state["a"], case["d"], case["marginal"]))
    if kind == "batch":
        values, index, _ = state["batch"].solve()
        return {"values": values, "gray_index": index}
    if kind == "learned":
        return [_solution(s) for s, _ in _learned().solve_learned_batch(state["mats"], state["proposer"])]
    grads, loss = state["net"].gradients(state["x"], state["t"], state["mask"])
    return {"loss": np.float32(loss), **grads}


# ---- what a pass cannot do without ---------------------------------------------

def _enumeration(rows, cols, d):
    """Operations of an exhaustive solve: one absolute value and one sum per
    column, message and labeling; labelings that differ by a permutation of the
    free messages count once."""
    base = 2 if d <= 2 else d
    return 2.0 * d * cols * base ** (rows - 1) / math.factorial(max(d - 1, 1))


def work(case):
    kind = case["kind"]
    if kind in ("text", "solve"):
        r, c = case["rows"], case["cols"]
        return {"bytes": 8 * r * c + 4 * r + 16, "flops": _enumeration(r, c, case["d"])}
    if kind == "batch":
        rows = range(16, case["max_rows"] + 1)
        each = sum(0.6 * _enumeration(n, 40, 1) + 0.3 * _enumeration(n, 40, 2) for n in rows) / len(rows)
        each += 0.05 * (_enumeration(16, 40, 3) + _enumeration(17, 40, 3))
        return {"bytes": case["count"] * (8 * 20 * 40 + 16), "flops": case["count"] * each}
    if kind == "learned":
        # the proposals' forward pass, one sweep of single-row moves over every
        # start, and a bound for each of 2^20 prefixes
        n, p = case["rows"], case["directions"]
        net = 2.0 * p * (44 * 256 + 256 * 256 + 256 * 44)
        return {"bytes": case["count"] * (8 * n * 44 + 4 * n + 16),
                "flops": case["count"] * (net + 2.0 * p * n * n * 44 + 2.0 * 44 * 2 ** 20)}
    rows, params = case["rows"], 44 * 256 + 256 * 256 + 256 * 44
    return {"bytes": 4 * (3 * rows * 44 + 2 * params + 2 * (256 + 256 + 44)), "flops": 6.0 * rows * params}


# ---- the same outputs in 64 bits, where they are quick to have --------------------

def _gray_labels(index, rows, d):
    """Labels of rows 0 .. rows-2 for Gray indices (the reflected base-d code)."""
    base = 2 if d <= 2 else d
    out = np.empty((len(index), rows - 1), dtype=np.int64)
    q = index.copy()
    for i in range(rows - 1):
        r = q % (2 * base)
        out[:, i] = np.where(r < base, r, 2 * base - 1 - r)
        q //= base
    return out


def _exact_solve(a, d, marginal):
    rows = a.shape[0]
    total = (2 if d <= 2 else d) ** (rows - 1)
    best, at = None, 0
    for n0 in range(0, total, 1 << 16):
        lab = _gray_labels(np.arange(n0, min(total, n0 + (1 << 16)), dtype=np.int64), rows, d)
        lab = np.concatenate([lab, np.full((len(lab), 1), 1 if d == 1 else 0, np.int64)], axis=1)
        if d == 1:
            s = (2 * lab - 1) @ a
            v = np.abs(s[:, 1:]).sum(1) + (s[:, 0] if marginal else np.abs(s[:, 0]))
        else:
            v = sum(np.abs((lab == m).astype(np.int64) @ a).sum(1) for m in range(d))
        i = int(np.argmax(v))
        if best is None or v[i] > best:
            best, at = int(v[i]), n0 + i
    return {"value": np.int64(best), "gray_index": np.uint64(at),
            "labels": _gray_labels(np.array([at], dtype=np.int64), rows, d)[0].astype(np.int32)}


def exact(case, seed):
    if case["kind"] == "solve":
        if _enumeration(case["rows"], case["cols"], case["d"]) * math.factorial(max(case["d"] - 1, 1)) > 2.0 ** 27:
            return None
        return _exact_solve(_matrix(case, np.random.default_rng(seed)), case["d"], case["marginal"])
    if case["kind"] != "gradient":
        return None
    params, x, t, mask = _net_inputs(case, seed)
    p = {k: v.astype(np.float64) for k, v in params.items()}
    x, t, mask = (v.astype(np.float64) for v in (x, t, mask))
    h1 = np.maximum(x @ p["W1"].T + p["b1"], 0.0)
    h2 = np.maximum(h1 @ p["W2"].T + p["b2"], 0.0)
    z = h2 @ p["W3"].T + p["b3"] + SKIP * x
    inv = 1.0 / mask.sum()
    loss = float((mask * (np.maximum(z, 0.0) - z * t + np.log1p(np.exp(-np.abs(z))))).sum() * inv)
    dz3 = (1.0 / (1.0 + np.exp(-z)) - t) * mask * inv
    dz2 = (dz3 @ p["W3"]) * (h2 > 0)
    dz1 = (dz2 @ p["W2"]) * (h1 > 0)
    return {"loss": loss, "W1": dz1.T @ x, "b1": dz1.sum(0), "W2": dz2.T @ h1, "b2": dz2.sum(0),
            "W3": dz3.T @ h2, "b3": dz3.sum(0)}
