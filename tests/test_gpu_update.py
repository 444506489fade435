"""Resident scenes and incremental updates (pbig2_scene_*): after every move
the scene's full pair list equals a fresh query of the moved boxes, and the
removed / added lists are exactly the pairs that involve a moved box before
and after the move."""
import numpy as np
import pytest

from oracle import oracle as O
from pbig_gb300 import PbigError, Scene, gen
from pbig_gb300.serve import move_indices

pytestmark = pytest.mark.gpu


def canon(p):
    return O.sort_pairs(np.asarray(p, dtype=np.uint32).reshape(-1, 2))


def touching(pairs, moved):
    m = np.zeros(int(max(pairs.max() if len(pairs) else 0, moved.max())) + 1, dtype=bool)
    m[moved] = True
    return canon(pairs[m[pairs[:, 0]] | m[pairs[:, 1]]]) if len(pairs) else canon(pairs)


@pytest.mark.parametrize("dims", [2, 3])
def test_moves_keep_the_pair_set_exact(engine, dims):
    boxes = gen.clustered3d(200000, seed=11) if dims == 3 else gen.uniform2d(100000, seed=5, side=(0.002, 0.01))
    if dims == 2:
        boxes = np.ascontiguousarray(boxes)
    sc = Scene(engine, boxes, gen.RANGE)
    try:
        cur = boxes.copy()
        before = canon(sc.pairs())
        assert sc.npairs == len(before)
        assert np.array_equal(before, O.grid_pairs(cur, gen.RANGE)[0])
        for step in range(6):
            idx = move_indices(len(cur), 0.01 if step % 2 == 0 else 0.05, 100 + step)
            nb = cur[idx].copy()
            if dims == 3:
                tmp = cur.copy()
                gen.move3d(tmp, idx, 7 + step, sigma=0.002)
                nb = tmp[idx]
            else:  # 2-D: shift by a seeded amount, clipped to the range
                rng = np.random.default_rng(step)
                d = rng.integers(-20000, 20000, size=(len(idx), 2))
                for a in range(2):
                    lo = np.clip(nb[:, 2 * a].astype(np.int64) + d[:, a], 0, gen.RANGE - 1)
                    w = nb[:, 2 * a + 1].astype(np.int64) - nb[:, 2 * a]
                    nb[:, 2 * a] = lo
                    nb[:, 2 * a + 1] = np.minimum(lo + w, gen.RANGE - 1)
            nr, na = sc.move(idx, nb)
            after_boxes = cur.copy()
            after_boxes[idx] = nb
            want = O.grid_pairs(after_boxes, gen.RANGE)[0]
            got = canon(sc.pairs())
            assert np.array_equal(got, want), step
            rem, add = sc.delta()
            assert nr == len(rem) and na == len(add)
            assert np.array_equal(canon(rem), touching(before, idx))
            assert np.array_equal(canon(add), touching(want, idx))
            cur, before = after_boxes, want
    finally:
        sc.close()


def test_slack_overflow_rebuilds_the_grid(engine):
    """Moving many boxes into one place overflows the slack of its cells; the
    grid is rebuilt and the results stay exact."""
    boxes = gen.scene3d(50000, seed=3)
    sc = Scene(engine, boxes, gen.RANGE, cell_shift=16)
    try:
        idx = np.arange(0, 50000, 10, dtype=np.uint32)
        nb = boxes[idx].copy()
        nb[:, [0, 2, 4]] = 5000000
        nb[:, [1, 3, 5]] = 5000000 + 1000
        nr, na = sc.move(idx, nb)
        cur = boxes.copy()
        cur[idx] = nb
        assert np.array_equal(canon(sc.pairs()), O.grid_pairs(cur, gen.RANGE)[0])
        assert na >= len(idx) * (len(idx) - 1) // 2  # all moved boxes are identical now
    finally:
        sc.close()


def test_bad_moves_are_refused(engine):
    boxes = gen.scene3d(20000, seed=4)
    sc = Scene(engine, boxes, gen.RANGE)
    try:
        idx = np.array([5, 9, 5], dtype=np.uint32)
        with pytest.raises(PbigError):
            sc.move(idx, boxes[idx])
        bad = boxes[[1, 2]].copy()
        bad[0, 0], bad[0, 1] = 100, 50  # min > max
        with pytest.raises(PbigError):
            sc.move(np.array([1, 2], dtype=np.uint32), bad)
        wrong = boxes[[1, 2]].copy()
        wrong[:, 6] = [2, 1]  # rid must be the index
        with pytest.raises(PbigError):
            sc.move(np.array([1, 2], dtype=np.uint32), wrong)
        # the scene is unchanged and still usable
        assert np.array_equal(canon(sc.pairs()), O.grid_pairs(boxes, gen.RANGE)[0])
        sc.move(np.array([3], dtype=np.uint32), boxes[[3]])
        assert np.array_equal(canon(sc.pairs()), O.grid_pairs(boxes, gen.RANGE)[0])
    finally:
        sc.close()


def test_delta_only_scene(engine):
    """PBIG2_SCENE_DELTA_ONLY: the moves report the same delta, no full list."""
    boxes = gen.clustered3d(100000, seed=12)
    sc = Scene(engine, boxes, gen.RANGE, keep_pairs=False)
    try:
        before = O.grid_pairs(boxes, gen.RANGE)[0]
        idx = move_indices(len(boxes), 0.02, 9)
        cur = boxes.copy()
        gen.move3d(cur, idx, 9, sigma=0.002)
        sc.move(idx, cur[idx])
        rem, add = sc.delta()
        after = O.grid_pairs(cur, gen.RANGE)[0]
        assert np.array_equal(canon(rem), touching(before, idx))
        assert np.array_equal(canon(add), touching(after, idx))
        with pytest.raises(PbigError):
            sc.pairs()
    finally:
        sc.close()


def shifted(boxes, idx, by, rng):
    """Rows idx moved by `by` along every axis, within the range."""
    nb = boxes[idx].astype(np.int64)
    dims = (boxes.shape[1] - 1) // 2
    for a in range(dims):
        w = nb[:, 2 * a + 1] - nb[:, 2 * a]
        nb[:, 2 * a] = np.clip(nb[:, 2 * a] + by[:, a], 0, rng - 1 - w)
        nb[:, 2 * a + 1] = nb[:, 2 * a] + w
    return nb.astype(np.uint32)


@pytest.mark.parametrize("keep_pairs", [True, False])
@pytest.mark.parametrize("dims,shift", [(2, 18), (3, 20), (3, 19)])
def test_moves_within_cells_and_out_of_them(engine, dims, shift, keep_pairs):
    """Boxes of 1 to hundreds of cells that stay in all their cells, in some of
    them or in none; few boxes and all; lists that grow beyond their buffers."""
    rs = np.random.default_rng(dims * 100 + shift)
    n, rng, cell = 20000, gen.RANGE, 1 << shift
    boxes = np.empty((n, 2 * dims + 1), dtype=np.uint32)
    for a in range(dims):
        side = np.where(np.arange(n) % 500 == 7, 7 * cell, rng // 400)
        lo = rs.integers(0, rng - side)
        boxes[:, 2 * a], boxes[:, 2 * a + 1] = lo, lo + rs.integers(0, side + 1)
    boxes[:, -1] = np.arange(n)
    sc = Scene(engine, boxes, rng, cell_shift=shift, keep_pairs=keep_pairs)
    try:
        cur, before = boxes.copy(), O.grid_pairs(boxes, rng)[0]
        for k, reach in [(1, 0), (33, 3), (500, cell // 50), (500, cell), (2000, rng // 3), (n, cell // 10), (40, 8 * cell)]:
            idx = rs.choice(n, k, replace=False).astype(np.uint32)
            idx[0] = 7 if 7 not in idx else idx[0]  # (a large box each time)
            nb = shifted(cur, idx, rs.integers(-reach, reach + 1, size=(k, dims)), rng)
            nr, na = sc.move(idx, nb)
            cur[idx] = nb
            after = O.grid_pairs(cur, rng)[0]
            rem, add = sc.delta()
            assert (nr, na) == (len(rem), len(add))
            assert np.array_equal(canon(rem), touching(before, idx)), (k, reach)
            assert np.array_equal(canon(add), touching(after, idx)), (k, reach)
            if keep_pairs:
                assert np.array_equal(canon(sc.pairs()), after), (k, reach)
            before = after
    finally:
        sc.close()


def test_a_refused_move_keeps_the_last_lists(engine):
    boxes = gen.scene3d(30000, seed=8)
    sc = Scene(engine, boxes, gen.RANGE)
    try:
        idx = np.arange(100, 200, dtype=np.uint32)
        sc.move(idx, shifted(boxes, idx, np.full((100, 3), 50000), gen.RANGE))
        lists = [canon(v) for v in sc.delta()] + [canon(sc.pairs())]
        many = np.arange(30000, dtype=np.uint32)  # (more room asked for than there is)
        bad = boxes.copy()
        bad[29999, 1] = gen.RANGE
        twice = many.copy()
        twice[5] = 6
        for i, b in ((many, bad), (twice, boxes[twice]), (np.array([30000], dtype=np.uint32), boxes[:1])):
            with pytest.raises(PbigError):
                sc.move(i, b)
            for want, got in zip(lists, [*sc.delta(), sc.pairs()]):
                assert np.array_equal(want, canon(got))
        nr, na = sc.move(many, boxes)
        assert nr == len(lists[2]) and np.array_equal(canon(sc.pairs()), O.grid_pairs(boxes, gen.RANGE)[0])
    finally:
        sc.close()


@pytest.mark.parametrize("dims", [2, 3])
@pytest.mark.parametrize("large", [0, 1])
def test_automatic_grids_of_scenes(engine, dims, large):
    """Automatic cell sizes, with the finer grid that small boxes get and, where
    a box covers most of the range, the query's."""
    rs = np.random.default_rng(dims + 10 * large)
    for n in (40, 7000):
        side = int(gen.RANGE * (1.0 / n) ** (1 / dims))
        boxes = np.empty((n, 2 * dims + 1), dtype=np.uint32)
        lo = rs.integers(0, gen.RANGE - side, size=(n, dims))
        boxes[:, 0:2 * dims:2], boxes[:, 1:2 * dims:2] = lo, lo + rs.integers(0, side, size=(n, dims))
        if large:
            boxes[n // 2, 0:2 * dims:2], boxes[n // 2, 1:2 * dims:2] = 0, gen.RANGE - 1
        boxes[:, -1] = np.arange(n)
        sc = Scene(engine, boxes, gen.RANGE)
        try:
            cur = boxes.copy()
            assert np.array_equal(canon(sc.pairs()), O.brute_pairs(cur))
            for step in range(3):
                idx = rs.choice(n, n // 3, replace=False).astype(np.uint32)
                idx[0] = n // 2 if n // 2 not in idx else idx[0]
                cur[idx] = shifted(cur, idx, rs.integers(-side, side + 1, size=(len(idx), dims)), gen.RANGE)
                sc.move(idx, cur[idx])
                assert np.array_equal(canon(sc.pairs()), O.brute_pairs(cur)), (n, step)
        finally:
            sc.close()
