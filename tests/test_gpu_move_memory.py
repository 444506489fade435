"""Moves of a resident scene that run out of device memory on the way: the scene
is what it was before the move, and the next one is exact."""
import numpy as np
import pytest

from oracle import oracle as O
from pbig_gb300 import Engine, PbigError, Scene
from pbig_gb300.engine import ENOMEM

pytestmark = pytest.mark.gpu
RANGE, N = 1 << 24, 30000


def scene(seed):
    r = np.random.default_rng(seed)
    side = RANGE // 50
    lo = r.integers(0, RANGE - side, size=(N, 3))
    b = np.empty((N, 7), dtype=np.uint32)
    b[:, 0:6:2], b[:, 1:6:2] = lo, lo + r.integers(0, side, size=(N, 3))
    b[:, 6] = np.arange(N)
    return b


def canon(p):
    return O.sort_pairs(np.asarray(p, dtype=np.uint32).reshape(-1, 2))


def touching(pairs, idx):
    return pairs[np.isin(pairs[:, 0], idx) | np.isin(pairs[:, 1], idx)]


def gather(b, idx):
    """All of idx at one place: pairs of each with each."""
    nb = b[idx].copy()
    nb[:, :6] = [RANGE // 2, RANGE // 2 + 9] * 3
    return nb


def widen(b, idx):
    """All of idx over half the range: many cells each, and pairs with an eighth of the boxes."""
    nb = b[idx].copy()
    nb[:, :6] = [1, RANGE // 2] * 3
    return nb


# list: the list of added pairs cannot grow; full: the full list cannot; grid:
# a cell overflows and the grid cannot be built anew
@pytest.mark.parametrize("keep_pairs", [True, False])
@pytest.mark.parametrize("what,change,limit", [("list", gather, 150 << 10), ("full", gather, 420 << 10), ("grid", widen, 420 << 10)])
def test_a_move_without_memory_changes_nothing(what, change, limit, keep_pairs):
    if what == "full" and not keep_pairs:
        pytest.skip("no full list is kept")
    boxes = scene(5)
    idx, other = np.arange(100, 400, dtype=np.uint32), np.arange(350, 700, dtype=np.uint32)
    with Engine(0) as engine:
        sc = Scene(engine, boxes, RANGE, cell_shift=20, keep_pairs=keep_pairs)
        try:
            for _ in range(2):  # (both full lists and the small buffers are there)
                sc.move(idx, boxes[idx])
            before = O.grid_pairs(boxes, RANGE)[0]
            assert 3000 < len(before) < 5000  # (what the limits are counted for)
            engine.set_max_buffer(limit)
            with pytest.raises(PbigError) as e:
                sc.move(idx, change(boxes, idx))
            assert e.value.code == ENOMEM
            assert [len(v) for v in sc.delta()] == [0, 0]
            if keep_pairs:
                assert np.array_equal(canon(sc.pairs()), before)
            engine.set_max_buffer(0)
            for moved, way in ((other, gather), (idx, change)):
                nb = way(boxes, moved)
                sc.move(moved, nb)
                boxes[moved] = nb
                after = O.grid_pairs(boxes, RANGE)[0]
                rem, add = sc.delta()
                assert np.array_equal(canon(rem), touching(before, moved))
                assert np.array_equal(canon(add), touching(after, moved))
                if keep_pairs:
                    assert np.array_equal(canon(sc.pairs()), after)
                before = after
        finally:
            sc.close()
