"""The tensor-core enumeration (tc_kernel.cuh), which large solves of matrices
with small entries take: bit-exact against the oracle (value and smallest
Gray index) for d = 1, LM, 2, 3 and 4, over column counts at the edges of the
byte words, +-1 entries (ties, both parities of a column's sum), entries to
+-3, one-sided columns, equal rows, zero columns, shards, label symmetry on
and off, repeated launches of a plan, and inside a batch."""
import contextlib

import numpy as np
import pytest

import oracle_ffi as O

pytestmark = pytest.mark.gpu

ROWS = {1: 27, 2: 27, 3: 17, 4: 14}


def _solve(ld, a, d, marg, **kw):
    plan = ld.Plan(a, d, marg, ld.options(**kw))
    desc = plan.describe()
    sol = plan.solve()
    plan.close()
    return sol, desc


def _tc(desc):
    return int(desc.split("tc=")[1].split()[0])


def _chunks(desc):
    """Chunks per tile (tc_chunk_steps); 0 without the tensor-core form."""
    steps = _tc(desc) // 16
    return 0 if steps == 0 else 1 if steps <= 16 else -(-steps // (12 if steps in (22, 24) else 10))


def _matrix(rng, d, cols, kind, rows=0):
    shape = (rows or ROWS[d], cols)
    if kind == "pm1":
        return rng.choice(np.array([-1, 1], dtype=np.int64), size=shape)
    if kind == "sparse":
        a = rng.integers(-1, 2, size=shape)
        a[:, cols // 2] = 0
        a[2] = a[1]
        return a.astype(np.int64)
    a = rng.integers(-3, 4, size=shape).astype(np.int64)
    a[:, -1] = np.abs(a[:, -1])
    return a


@pytest.mark.parametrize("kind", ["pm1", "sparse", "amp3"])
@pytest.mark.parametrize("d,marg,cols", [(1, False, 9), (1, False, 16), (1, False, 33), (1, True, 37), (1, True, 48),
                                         (2, False, 11), (2, False, 16), (2, False, 24), (3, False, 10),
                                         (3, False, 17), (3, False, 30), (4, False, 8), (4, False, 21)])
def test_matches_the_oracle(ld, d, marg, cols, kind):
    rng = np.random.default_rng(100 * d + cols + len(kind))
    a = _matrix(rng, d, cols, kind)
    if marg:
        a[:, 0] = rng.integers(-5, 6, size=a.shape[0])
    ref = O.enumerate_max(a, d, marg)
    sol, desc = _solve(ld, a, d, marg)
    assert _tc(desc) > 0 or kind == "amp3" or cols < 12, desc
    assert (sol.value, sol.gray_index) == ref, desc
    table, desc = _solve(ld, a, d, marg, paired_walks=-1)
    assert _tc(desc) == 0 and (table.value, table.gray_index) == ref, desc
    assert sol.evaluated <= sol.labelings == table.labelings


@pytest.mark.parametrize("d,rows,cols", [(1, 28, 36), (3, 18, 28)])
def test_shards_launches_and_every_walk(ld, d, rows, cols):
    rng = np.random.default_rng(rows)
    a = _matrix(rng, d, cols, "pm1", rows)
    ref = O.enumerate_max(a, d, False)
    plan = ld.Plan(a, d)
    assert _tc(plan.describe()) > 0, plan.describe()
    whole = plan.solve()
    for _ in range(3):
        again = plan.solve()
        assert (again.value, again.gray_index) == (whole.value, whole.gray_index) == ref
    plan.close()
    best, lo, work = None, 0, 0
    for i in range(2):
        plan = ld.Plan(a, d, False, ld.options(shard_index=i, shard_count=2))
        assert plan.range[0] == lo
        lo = plan.range[1]
        sol = plan.solve()
        plan.close()
        cand = (sol.value, -sol.gray_index)
        best = cand if best is None or cand > best else best
        work += sol.evaluated
    assert lo == O.total(rows, d) and (best[0], -best[1]) == ref
    if d >= 3:
        full, desc = _solve(ld, a, d, False, enumerate_all=1)
        assert _tc(desc) > 0 and (full.value, full.gray_index) == ref
        assert whole.evaluated < full.evaluated == full.labelings


def test_a_block_of_ties(ld):
    """Every labeling of the low rows ties: the smallest index is reported."""
    a = np.zeros((28, 40), dtype=np.int64)
    a[:, :20] = 1
    a[12:, 20:] = np.random.default_rng(3).choice([-1, 1], size=(16, 20))
    a[:12, :20] = 0
    a[:12, 20] = 1
    ref = O.enumerate_max(a, 1, False)
    sol, desc = _solve(ld, a, 1, False)
    assert (sol.value, sol.gray_index) == ref, desc


@pytest.mark.parametrize("rows", [38, 39, 40])
def test_at_most_32_high_rows_with_three_labels(ld, rows):
    """The kernel keeps a walk's labels in 64 bits, two per high row: more than
    32 high rows stay with the table kernel.  (With 33 and 34 high rows, shards
    beyond the first third of the range reported values that their labels do
    not have: 152 for 88.)  The plans are only described: such a shard is long."""
    a = _matrix(np.random.default_rng(rows), 3, 12, "pm1", rows)
    for index in (0, 2 ** 30, 2 ** 31 - 2):
        plan = ld.Plan(a, 3, False, ld.options(shard_index=index, shard_count=2 ** 31 - 1))
        desc = plan.describe()
        plan.close()
        assert (_tc(desc) > 0) == (rows - 1 - 5 <= 32), desc


@pytest.mark.parametrize("d,marg,cols,chunks", [(1, False, 16, 1), (1, False, 33, 2), (1, True, 48, 3), (2, False, 16, 1),
                                                (2, False, 24, 2), (3, False, 17, 1), (3, False, 30, 3), (4, False, 21, 2)])
def test_a_wait_that_runs_out(ld, d, marg, cols, chunks):
    """Waits that give up at once: the plan and the one-shot solve fail with
    LD_ERR_TIMEOUT, and the next solves are right.  Waits of one poll may run
    out anywhere: the solve fails in the same way or is right."""
    a = _matrix(np.random.default_rng(cols), d, cols, "pm1")
    ref = O.enumerate_max(a, d, marg)
    good = ld.Plan(a, d, marg)
    assert _chunks(good.describe()) == chunks, good.describe()
    for polls in (-1, 1):
        plan = ld.Plan(a, d, marg, ld.options(wait_polls=polls))
        for solve in (plan.solve, plan.solve, lambda: ld.solve_reduced(a, d, marg, ld.options(wait_polls=polls))):
            try:
                sol = solve()
                assert polls == 1 and (sol.value, sol.gray_index) == ref
            except ld.LdError as e:
                assert e.status == 7
            sol = good.solve()
            assert (sol.value, sol.gray_index) == ref
        plan.close()
    good.close()
    sol = ld.solve_reduced(a, d, marg)
    assert (sol.value, sol.gray_index) == ref
    with pytest.raises(ld.LdError) as e:
        ld.Plan(a, d, marg, ld.options(wait_polls=-2))
    assert e.value.status == 1


@contextlib.contextmanager
def ld_batch(ld, mats, ds, tune, **kw):
    b = ld.Batch(mats, ds, opts=ld.options(**kw), autotune=tune)
    try:
        yield b
    finally:
        b.close()


@pytest.mark.parametrize("tune", [False, True])
def test_inside_a_batch(ld, tune):
    """Batch entries that get their own plan take the tensor-core form too; a
    wait that runs out there fails the batch instead of being its value."""
    rng = np.random.default_rng(44)
    mats = [_matrix(rng, 4, 21, "pm1"), rng.integers(-90, 91, size=(12, 20)).astype(np.int64), _matrix(rng, 4, 8, "amp3"),
            _matrix(rng, 4, 20, "pm1", 11)]
    ds = [4, 1, 4, 4]
    refs = [O.enumerate_max(a, d, False) for a, d in zip(mats, ds)]
    assert _tc(_solve(ld, mats[0], 4, False)[1]) > 0
    with ld_batch(ld, mats, ds, tune) as b:
        for _ in range(2):
            v, g, _ = b.solve()
            assert [(int(x), int(y)) for x, y in zip(v, g)] == refs, b.describe()
    with ld_batch(ld, mats, ds, tune, wait_polls=-1) as b:
        for _ in range(2):
            with pytest.raises(ld.LdError) as e:
                b.solve()
            assert e.value.status == 7 and "entry 0" in str(e.value)


@pytest.mark.parametrize("d,cols,amp,seed,chunks", [(1, 17, 3, 24, 1), (1, 20, 3, 27, 2), (2, 10, 3, 24, 1), (2, 11, 3, 25, 2),
                                                    (2, 15, 3, 29, 3), (3, 15, 2, 36, 1), (3, 15, 3, 36, 2), (3, 18, 3, 39, 3),
                                                    (4, 17, 2, 45, 1), (4, 17, 3, 45, 2), (4, 17, 3, 17, 3)])
def test_weights_above_one_in_every_number_of_chunks(ld, d, cols, amp, seed, chunks):
    """Entries to +-2 and +-3: thresholds that share a feature, in tiles of one,
    two and three chunks for every order (+-1 entries reach three chunks for d = 1
    and 3 alone)."""
    a = np.random.default_rng(seed).integers(-amp, amp + 1, size=(ROWS[d], cols)).astype(np.int64)
    sol, desc = _solve(ld, a, d, False)
    assert _chunks(desc) == chunks, desc
    assert (sol.value, sol.gray_index) == O.enumerate_max(a, d, False), desc


@pytest.mark.parametrize("d,cols", [(1, 40), (2, 24), (3, 30), (4, 21)])
def test_every_low_labeling_of_a_block_ties(ld, d, cols):
    """Rows of the table that are zero: all labelings of a block have its value,
    and the block's first Gray index is the one reported."""
    low = {1: 8, 2: 8, 3: 5, 4: 4}[d]
    for seed in range(4):
        a = np.random.default_rng(seed).choice(np.array([-1, 1], dtype=np.int64), size=(ROWS[d], cols))
        a[:low] = 0
        sol, desc = _solve(ld, a, d, False)
        assert _tc(desc) > 0 and f" k={low} " in desc, desc
        assert (sol.value, sol.gray_index) == O.enumerate_max(a, d, False), desc
        assert sol.gray_index % (2 if d <= 2 else d) ** low == 0
