"""The order of the tensor-core kernel's shared-memory slots (no GPU): every
slot that its producers use again has been read by the epilogue before, for
tiles of one, two and three chunks and walks of one high index and more.

A set's producers, its matrix warp and its epilogue are three sequences of
events; the barriers add edges between them (the rules are those of
tc_kernel.cuh's `take`, `commit` and waits).  Where the epilogue reads each
array, before or after it releases the tile's accumulators, is taken from the
source."""
import re
from pathlib import Path

import pytest

KERNEL = Path(__file__).resolve().parents[1] / "l-norms_bruteforce_b200" / "csrc" / "kernels" / "tc_kernel.cuh"
SLOTS = 4
TILES = 24


def _epilogue_order():
    """{array: it is read before the release of the accumulators}"""
    code = re.sub(r"//[^\n]*", "", KERNEL.read_text().split("---- epilogue")[1].split("__syncthreads()")[0])
    release = code.index("bar_arrive(&acc_empty[g])")
    reads = {name: [m.start() for m in re.finditer(rf"\b{name}\[g\]", code)] for name in ("s_base", "s_where", "s_high")}
    assert all(reads.values()), reads
    return {name: max(at) < release for name, at in reads.items()}


def _unordered(chunks, walk_len, read_early):
    """(array, tile that reads, tile that overwrites) without an order."""
    before = {}                                     # event -> events that must precede it

    def chain(events):
        for a, b in zip(events, events[1:]):
            before.setdefault(b, []).append(a)

    def edge(a, b):
        before.setdefault(b, []).append(a)

    produce, multiply, read = [], [], []
    for t in range(TILES):
        if t % walk_len == 0:
            produce.append(("write", "s_high", t))
        for n in range(chunks):
            c = t * chunks + n
            if c >= 2:                              # take(): the products of chunk c - 2 are done
                edge(("done", c - 2), ("take", c))
            produce.append(("take", c))
            if n == 0:
                produce += [("write", "s_base", t), ("write", "s_where", t), ("slot", t)]
            produce.append(("hand", c))
            edge(("hand", c), ("issue", c))
            multiply.append(("issue", c))
            edge(("issue", c), ("done", c))         # not in program order: the commit is asynchronous
            if c:
                edge(("done", c - 1), ("done", c))
        if t:
            edge(("release", t - 1), ("issue", t * chunks))
        early = [("read", name, t) for name, e in read_early.items() if e]
        late = [("read", name, t) for name, e in read_early.items() if not e]
        edge(("slot", t), ("look", t))
        edge(("done", t * chunks + chunks - 1), ("load", t))
        read += [("look", t)] + early + [("load", t), ("release", t)] + late
    for seq in (produce, multiply, read):
        chain(seq)

    def precedes(a, b):
        seen, todo = set(), [b]
        while todo:
            e = todo.pop()
            if e == a:
                return True
            if e not in seen:
                seen.add(e)
                todo += before.get(e, [])
        return False

    bad = []
    for t in range(TILES):
        for name, unit in (("s_base", 1), ("s_where", 1), ("s_high", walk_len)):
            over = (t // unit + SLOTS) * unit       # the tile whose producers write the same slot next
            if over < TILES and not precedes(("read", name, t), ("write", name, over)):
                bad.append((name, t, over))
    return bad


@pytest.mark.parametrize("walk_len", [1, 2, 3, 4])
@pytest.mark.parametrize("chunks", [1, 2, 3])
def test_slots_are_read_before_they_are_used_again(chunks, walk_len):
    assert not _unordered(chunks, walk_len, _epilogue_order())


def test_the_model_sees_a_late_read():
    """Walks of one high index, one chunk per tile, the group's walks read
    after the release: the producers may be past it."""
    late = {"s_base": True, "s_where": True, "s_high": False}
    assert {b[0] for b in _unordered(1, 1, late)} == {"s_high"}
    assert not _unordered(2, 1, late) and not _unordered(1, 2, late)
