"""Pruned search over several levels of prefixes and over several launches of
high indices, and the local search's two integer widths: the answers are those
of the plain enumeration (itself checked against the oracle) and of the same
moves made one by one in Python."""
import time

import numpy as np
import pytest

import oracle_ffi as O

pytestmark = pytest.mark.gpu


def _matrix(rng, rows, cols, kind):
    if kind == "lowrank":
        a = 5 * rng.standard_normal((rows, 3)) @ rng.standard_normal((3, cols))
        return np.rint(a).astype(np.int64) + rng.integers(-1, 2, size=(rows, cols))
    return rng.integers(-kind, kind + 1, size=(rows, cols)).astype(np.int64)


@pytest.mark.parametrize("rows,cols,d,marg,kind", [
    (38, 44, 1, False, "lowrank"),   # 32-bit lanes, an extended level
    (36, 40, 1, True, "lowrank"),
    (34, 12, 1, False, 1),           # 8-bit lanes
    (33, 17, 2, False, "lowrank"),
    (34, 9, 2, False, 1),
    (21, 13, 3, False, "lowrank"),
    (12, 64, 1, False, 40),          # a single prefix
])
def test_levels(ld, rows, cols, d, marg, kind):
    rng = np.random.default_rng(rows * 100 + cols)
    a = _matrix(rng, rows, cols, kind)
    plain = ld.solve_reduced(a, d, marg)
    vals, labs = ld.local_search(a, d, marg, n_random=16, seed=2)
    for lab in (labs[int(np.argmax(vals))], labs[int(np.argmin(vals))], O.labels(plain.gray_index, rows, d)):
        sol, st = ld.solve_pruned(a, d, marg, lab, ld.options(prune_policy=1))
        assert (sol.value, sol.gray_index) == (plain.value, plain.gray_index), st
        assert st["pruned"] == 1 and st["highs_kept"] <= st["highs_visited"] <= st["highs_total"]


@pytest.mark.parametrize("rows,cols,d", [(32, 7, 1), (31, 5, 2), (19, 4, 3)])
def test_everything_survives(ld, rows, cols, d):
    """Without an incumbent nothing is dropped: the high indices are bounded
    and evaluated in several launches."""
    a = _matrix(np.random.default_rng(rows), rows, cols, 9)
    plain = ld.solve_reduced(a, d)
    sol, st = ld.solve_pruned(a, d, False, None, ld.options(prune_policy=1, enumerate_all=1))
    assert (sol.value, sol.gray_index) == (plain.value, plain.gray_index)
    assert st["highs_kept"] == st["highs_visited"] == st["highs_total"]


@pytest.mark.parametrize("rows,cols", [(14, 16), (12, 64)])
def test_reported_device_time_is_the_launches(ld, rows, cols):
    """bound_ms and scan_ms hold the search's launches, not the host's waits and
    the solve of the low rows between them, which alone takes longer than the
    bound and the evaluation of one walk (two short launches)."""
    a = _matrix(np.random.default_rng(rows * 100 + cols), rows, cols, 300)
    vals, labs = ld.local_search(a, 1, False, n_random=16, seed=2)
    lab, scan, norm = labs[int(np.argmax(vals))], [], []
    for _ in range(20):
        sol, st = ld.solve_pruned(a, 1, False, lab, ld.options(prune_policy=1))
        assert st["pruned"] == 1 and sol.kernel_ms == pytest.approx(st["bound_ms"] + st["scan_ms"])
        assert 0 < st["bound_ms"] and 0 < st["scan_ms"]
        scan.append(st["scan_ms"])
    low = np.concatenate([a[:st["low_rows"]], np.zeros((1, cols), np.int64)])
    for _ in range(20):
        t0 = time.perf_counter()
        ld.solve_reduced(low, 1)
        norm.append((time.perf_counter() - t0) * 1e3)
    assert min(scan) < min(norm)


@pytest.mark.parametrize("rows", [14, 33])
def test_reported_upload_holds_the_levels(ld, rows):
    """d = 2 uploads the prefix rows' column totals (16 words) for every level,
    d = 1 the image alone, which has the same size."""
    a = _matrix(np.random.default_rng(rows), rows, 16, "lowrank") * 100
    sent = []
    for d in (1, 2):
        vals, labs = ld.local_search(a, d, False, n_random=16, seed=1)
        sol, st = ld.solve_pruned(a, d, False, labs[int(np.argmax(vals))], ld.options(prune_policy=1))
        assert st["pruned"] == 1
        sent.append(sol.h2d_bytes)
    assert sent[1] > sent[0] and (sent[1] - sent[0]) % 64 == 0


def _climb(a, d, marg, lab):
    """Steepest single-row moves; ties to the smallest row, then label."""
    lab = list(lab)
    while True:
        now, best = O.value(a, d, marg, lab), None
        for i in range(len(lab)):
            for t in range(2 if d == 1 else d):
                if t == lab[i]:
                    continue
                g = O.value(a, d, marg, lab[:i] + [t] + lab[i + 1:]) - now
                if g > 0 and (best is None or g > best[0]):
                    best = (g, i, t)
        if best is None:
            return now, lab
        lab[best[1]] = best[2]


@pytest.mark.parametrize("scale", [1, 10 ** 9])   # int32 and int64 sums
@pytest.mark.parametrize("rows,cols,d,marg", [(2, 1, 1, False), (9, 33, 1, True), (17, 16, 2, False), (13, 20, 3, False)])
def test_local_search_moves(ld, rows, cols, d, marg, scale):
    rng = np.random.default_rng(rows)
    a = rng.integers(-3, 4, size=(rows, cols)).astype(np.int64) * scale
    starts = rng.integers(0, 2 if d == 1 else d, size=(5, rows - 1))
    vals, labs = ld.local_search(a, d, marg, starts=starts)
    for s, v, lab in zip(starts, vals, labs):
        assert (int(v), lab.tolist()) == _climb(a, d, marg, [int(x) for x in s])
