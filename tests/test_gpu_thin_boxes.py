"""Boxes whose sides are shorter than a scaled step of their cell, down to
points: each ties with itself in the tile tests, and with its like. In cells
narrower and wider than 2^15, of sizes at the edges of the tiles; whole numbers,
equal to brute force."""
import numpy as np
import pytest

from oracle import oracle as O
from pbig_gb300 import Engine

pytestmark = pytest.mark.gpu

SIZES = [2, 5, 6, 9, 25, 32, 33, 40, 63, 65, 96, 128, 129, 300, 512, 513, 600]


@pytest.fixture(scope="module")
def engines():
    one, many = Engine(0), Engine(0)
    many.set_one_launch(False)
    yield one, many
    one.close()
    many.close()


def thin(n, dims, shift, side, places, seed):
    """n boxes of at most `side` along every axis in one cell, some at the same
    places, some a coordinate apart, some across the cell's edges."""
    r = np.random.default_rng(seed)
    cell = 1 << shift
    at = r.integers(0, cell, size=(places, dims))[r.integers(0, places, size=n)]
    lo = cell + at + r.integers(0, 2, size=(n, dims)) - (r.random((n, dims)) < 0.05) * side
    hi = lo + r.integers(0, side + 1, size=(n, dims))
    rows = np.empty((n, 2 * dims + 1), dtype=np.uint32)
    rows[:, 0:2 * dims:2], rows[:, 1:2 * dims:2] = lo, hi
    rows[:, -1] = np.arange(n)
    return rows, 4 * cell


def canon(p):
    return O.sort_pairs(np.asarray(p, dtype=np.uint32).reshape(-1, 2))


@pytest.mark.parametrize("dims", [2, 3])
@pytest.mark.parametrize("shift,side", [(12, 0), (15, 0), (15, 2), (19, 0), (19, 20), (29, 0), (29, 3 << 14)])
def test_cells_of_thin_boxes(engines, dims, shift, side):
    for n in SIZES:
        for places in (n // 3 + 1, 4 * n):  # (most of them shared, and most of them alone)
            boxes, rng = thin(n, dims, shift, side, places, n + shift)
            want = O.brute_pairs(boxes)
            for e in engines:
                for _ in range(2):
                    assert e.self_intersect(boxes, rng, cell_shift=shift) == len(want), (n, places)
                    assert np.array_equal(canon(e.pairs()), want), (n, places)


@pytest.mark.parametrize("side", [0, 1, 64])
def test_scenes_of_thin_boxes(side):
    r = np.random.default_rng(side)
    n, rng = 150000, 1 << 24
    lo = r.integers(0, rng - 64, size=(n, 3))
    lo[1::3] = lo[0::3]
    b = np.empty((n, 7), dtype=np.uint32)
    b[:, 0:6:2], b[:, 1:6:2] = lo, lo + r.integers(0, side + 1, size=(n, 3))
    b[:, 6] = np.arange(n)
    want = O.grid_pairs(b, rng, cs=1 << 18)[0]
    with Engine(0) as e:
        assert e.self_intersect(b, rng) == len(want) >= n // 3
        assert np.array_equal(canon(e.pairs()), want)
