"""Grids of resident scenes that do not fit: boxes so small against their
spacing that the slots of the query's grid cannot all be numbered, and too
little memory for the finer grid that scenes get."""
import numpy as np
import pytest

from oracle import oracle as O
from pbig_gb300 import Engine, PbigError, Scene
from pbig_gb300.engine import ECAPACITY

pytestmark = pytest.mark.gpu
RANGE = 1 << 24
SIDE = 2048


def sparse(n, seed):
    """n boxes of side SIDE, every tenth beside the one before it."""
    r = np.random.default_rng(seed)
    lo = r.integers(0, RANGE - 4 * SIDE, size=(n, 3))
    lo[1::10] = lo[0::10][: len(lo[1::10])] + r.integers(0, SIDE, size=(len(lo[1::10]), 3))
    b = np.empty((n, 7), dtype=np.uint32)
    b[:, 0:6:2], b[:, 1:6:2] = lo, lo + SIDE - 1
    b[:, 6] = np.arange(n)
    return b


def canon(p):
    return O.sort_pairs(np.asarray(p, dtype=np.uint32).reshape(-1, 2))


def want(b):
    return O.grid_pairs(b, RANGE, cs=1 << 18)[0]


@pytest.mark.parametrize("n,one_launch", [(20000, False), (300000, True)])
def test_sparse_scenes_get_a_grid_that_fits(n, one_launch):
    boxes = sparse(n, n)
    with Engine(0) as engine:
        engine.set_one_launch(one_launch)
        sc = Scene(engine, boxes, RANGE)
        try:
            assert np.array_equal(canon(sc.pairs()), want(boxes))
            r = np.random.default_rng(1)
            for _ in range(2):
                idx = np.sort(r.choice(n, n // 50, replace=False)).astype(np.uint32)
                by = r.integers(0, SIDE, size=(len(idx), 3))
                boxes[idx, 0:6:2] += by.astype(np.uint32)
                boxes[idx, 1:6:2] += by.astype(np.uint32)
                sc.move(idx, boxes[idx])
                assert np.array_equal(canon(sc.pairs()), want(boxes))
        finally:
            sc.close()


def test_a_given_size_that_does_not_fit_is_refused():
    boxes = sparse(1000, 3)
    with Engine(0) as engine:
        with pytest.raises(PbigError) as e:
            Scene(engine, boxes, RANGE, cell_shift=14)  # 2^30 cells
        assert e.value.code == ECAPACITY
        sc = Scene(engine, boxes, RANGE, cell_shift=17)
        assert np.array_equal(canon(sc.pairs()), want(boxes))
        sc.close()


def test_without_memory_for_the_finer_grid_a_scene_keeps_the_querys():
    n, limit = 300000, 40 << 20
    r = np.random.default_rng(4)
    side = 0.6 * n ** (-1 / 3) * RANGE
    boxes = np.empty((n, 7), dtype=np.uint32)
    boxes[:, 0:6:2] = lo = r.integers(0, RANGE - int(side), size=(n, 3))
    boxes[:, 1:6:2] = lo + r.integers(0, int(side), size=(n, 3))
    boxes[:, 6] = np.arange(n)
    with Engine(0) as engine:
        engine.self_intersect(boxes, RANGE)
        cells = engine.stats()["cells"]
        assert 8 * cells <= 4 * n and 32 * (8 * cells * 4 + n + n // 2) > limit  # one size finer: taken, and too many slots
    with Engine(0) as engine:
        engine.set_max_buffer(limit)
        sc = Scene(engine, boxes, RANGE)
        try:
            idx = np.arange(0, n, 50, dtype=np.uint32)
            nb = boxes[idx].copy()
            nb[:, :6] = boxes[(idx + 25) % n, :6]
            sc.move(idx, nb)
            boxes[idx] = nb
            assert np.array_equal(canon(sc.pairs()), want(boxes))
        finally:
            sc.close()
