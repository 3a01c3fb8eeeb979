"""Two columns per 32-bit word (half_kernel.cuh): the kernels of d = 1, LM, 2
and 3 for matrices with large entries.  Bit-exact against the oracle (value
and smallest Gray index) at the edges of the word counts and of the column
split, at the largest values a field and a half of the packed accumulator can
hold, with one and two high indices per thread, shards, ties and label
symmetry; and in batches."""
import numpy as np
import pytest

import oracle_ffi as O

pytestmark = pytest.mark.gpu

ROWS = {1: 14, 2: 13, 3: 9}
KINDS = {"L1": (1, False), "LM": (1, True), "d2": (2, False), "d3": (3, False)}


def _solve(ld, a, d, marg, **kw):
    plan = ld.Plan(a, d, marg, ld.options(**kw))
    desc = plan.describe()
    sol = plan.solve()
    plan.close()
    return sol, desc


def _half(desc):
    return int(desc.split("half=")[1].split()[0])


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("cols", [2, 3, 4, 5, 8, 15, 20, 21, 43, 44, 61, 63, 64, 65, 97, 128, 129, 200, 255, 256])
def test_widths_match_the_oracle(ld, kind, cols):
    d, marg = KINDS[kind]
    rng = np.random.default_rng(1000 * d + 10 * cols + marg)
    a = rng.integers(-300, 301, size=(ROWS[d], cols)).astype(np.int64)
    a[3] = a[1]                                  # equal rows: tied labelings
    ref = O.enumerate_max(a, d, marg)
    sol, desc = _solve(ld, a, d, marg)
    # the 32-bit form stays where it has hardly more words, and where a half
    # of the packed accumulator could pass 65535 (63 columns x 14 rows x 300)
    assert _half(desc) > 0 or cols <= 5 or (d == 1 and cols in (63, 64)), desc
    assert (" split=0" in desc) == (cols <= 64), desc
    assert (sol.value, sol.gray_index) == ref, desc
    old, desc = _solve(ld, a, d, marg, pack16=-1)
    assert _half(desc) == 0 and (old.value, old.gray_index) == ref, desc


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("cols", [30, 64, 90, 180])
@pytest.mark.parametrize("low_rows", [0, 1, 4])
def test_one_and_two_high_indices_shards_and_fixed_walks(ld, kind, cols, low_rows):
    d, marg = KINDS[kind]
    rng = np.random.default_rng(d + cols + low_rows)
    a = rng.integers(-90, 91, size=(ROWS[d] + 1, cols)).astype(np.int64)
    a[:, 0] = 200                                # a column of one sign
    ref = O.enumerate_max(a, d, marg)
    for kw in (dict(blocks=1), dict(blocks=1, paired_walks=-1), dict(blocks=2, walk_fetch=-1), dict(tile=2, blocks=3)):
        sol, desc = _solve(ld, a, d, marg, low_rows=low_rows, **kw)
        assert _half(desc) > 0, desc
        assert (sol.value, sol.gray_index) == ref, (kw, desc)
    best = None
    for i in range(3):
        sol, desc = _solve(ld, a, d, marg, low_rows=low_rows, shard_index=i, shard_count=3)
        cand = (sol.value, -sol.gray_index)
        best = cand if best is None or cand > best else best
    assert (best[0], -best[1]) == ref


@pytest.mark.parametrize("kind", KINDS)
def test_field_and_accumulator_limits(ld, kind):
    """Entries scaled up until the form no longer fits: the answer is the
    oracle's on both sides of the line, and the line is met."""
    d, marg = KINDS[kind]
    seen = set()
    for cols in (3, 12, 40):
        for amp in (500, 1500, 3000, 5000, 9000, 20000):
            rng = np.random.default_rng(amp + cols)
            a = rng.integers(amp // 2, amp + 1, size=(ROWS[d] - 1, cols)) * rng.choice([-1, 1], size=(ROWS[d] - 1, cols))
            a = a.astype(np.int64)
            if amp % 3 == 0:
                a = np.abs(a)                    # every field at the end of its range
            sol, desc = _solve(ld, a, d, marg)
            assert (sol.value, sol.gray_index) == O.enumerate_max(a, d, marg), (amp, cols, desc)
            seen.add(_half(desc) > 0)
    assert seen == {True, False}


def test_batch_matches_the_oracle(ld):
    rng = np.random.default_rng(41)
    mats, ds, ms = [], [], []
    for t in range(48):
        d = 1 + t % 3
        a = rng.integers(-250, 251, size=(int(rng.integers(2, ROWS[d] + 1)), int(rng.integers(1, 65))))
        if t % 5 == 0:
            a[1] = a[0]
        if t % 7 == 0:
            a = a * 20000                         # too large for the 16-bit fields
        mats.append(a.astype(np.int64)); ds.append(d); ms.append(int(d == 1 and t % 2 == 0))
    for tune in (False, True):
        b = ld.Batch(mats, ds, ms, autotune=tune)
        desc = b.describe()
        v, g, _ = b.solve()
        b.close()
        assert "int16x2=28" in desc, desc
        for p, (a, d, m) in enumerate(zip(mats, ds, ms)):
            assert (int(v[p]), int(g[p])) == O.enumerate_max(a, d, bool(m)), (p, a.shape, d, m, desc)
