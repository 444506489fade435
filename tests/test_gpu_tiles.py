"""The pair kernels' tiles and 15-bit entry terms at their edges.

Every box of a scene lies in one cell of 2^shift, so a cell of n boxes goes to
the kernel of its class (lane groups up to 32 boxes, a warp up to 128, a team
up to 512, tile tasks above). Corners lie on a lattice: boxes that touch and
boxes one coordinate apart are as common as boxes that overlap, and in cells of
2^15 or wider many corners share one scaled term, so the tiles are tested again
on the whole coordinates. Whole numbers: equal to brute force, no tolerance.
"""
import numpy as np
import pytest

from oracle import oracle as O
from pbig_gb300 import Engine

pytestmark = pytest.mark.gpu

SIZES = [2, 4, 5, 31, 32, 33, 40, 63, 64, 65, 96, 97, 128, 129, 160, 257, 511, 512, 513, 600]


@pytest.fixture(scope="module")
def engines():
    one, many = Engine(0), Engine(0)
    many.set_one_launch(False)
    yield one, many
    one.close()
    many.close()


def lattice(n, dims, shift, step, seed):
    """n boxes inside the second cell along every axis (and some that reach out
    of it), corners on multiples of `step`, off by one now and then."""
    rs = np.random.default_rng(seed)
    cell = 1 << shift
    rng = min(4 * cell, (1 << 32) - 1)
    k = max(2, cell // step)
    lo = rs.integers(0, k, size=(n, dims)) * step + rs.integers(0, 2, size=(n, dims))
    hi = lo + rs.integers(0, max(2, k // 3), size=(n, dims)) * step + rs.integers(-1, 2, size=(n, dims))
    lo, hi = np.minimum(lo, hi), np.maximum(lo, hi)
    lo, hi = lo + cell - (rs.random((n, dims)) < 0.2) * step, hi + cell
    rows = np.empty((n, 2 * dims + 1), dtype=np.uint32)
    rows[:, 0:2 * dims:2] = np.clip(lo, 0, rng - 1)
    rows[:, 1:2 * dims:2] = np.clip(hi, 0, rng - 1)
    rows[:, -1] = np.arange(n)
    return rows, rng


def canon(p):
    return O.sort_pairs(np.asarray(p, dtype=np.uint32).reshape(-1, 2))


@pytest.mark.parametrize("dims", [2, 3])
@pytest.mark.parametrize("shift,step", [(6, 1), (14, 1 << 9), (15, 1), (15, 1 << 11), (16, 2), (20, 1 << 16), (30, 1 << 26)])
def test_cells_of_every_size(engines, dims, shift, step):
    for n in SIZES:
        boxes, rng = lattice(n, dims, shift, step, seed=n + 1000 * shift + dims)
        want = O.brute_pairs(boxes)
        for e in engines:
            for _ in range(2):  # (a first result too large for a launch's buffers is redone)
                assert e.self_intersect(boxes, rng, cell_shift=shift) == len(want), n
                assert np.array_equal(canon(e.pairs()), want), n


@pytest.mark.parametrize("dims", [2, 3])
@pytest.mark.parametrize("shift,step", [(6, 1), (15, 1 << 11), (20, 1 << 16), (30, 1 << 26)])
def test_two_colours_in_one_cell(engines, dims, shift, step):
    """Red/blue cells from one colour alone to halves, each colour's tiles
    full, one short and one over."""
    e = engines[1]
    for n, red in [(33, 1), (40, 0), (40, 40), (64, 32), (65, 33), (97, 31), (128, 64), (128, 127), (129, 1), (300, 65),
                   (512, 32), (512, 479), (600, 300)]:
        boxes, rng = lattice(n, dims, shift, step, seed=n + 7 * red + shift)
        want = O.brute_pairs(boxes)
        want = want[(want[:, 0] < red) & (want[:, 1] >= red)].astype(np.int64)
        want[:, 1] -= red
        blue = boxes[red:].copy()
        blue[:, -1] -= np.uint32(red)
        assert e.bipartite_intersect(boxes[:red].copy(), blue, rng, cell_shift=shift) == len(want), (n, red)
        got = e.pairs().astype(np.int64)
        assert np.array_equal(got[np.lexsort((got[:, 1], got[:, 0]))], want), (n, red)


@pytest.mark.parametrize("n", [64, 100, 128, 300, 512, 600])
@pytest.mark.parametrize("hits", [1, 11, 12, 13, 32, 63, 64])
def test_rows_of_many_pairs(engines, n, hits):
    """Boxes apart from one another, and every 20th of them a wide one that
    overlaps `hits` others: rows below, at and above the length that the warp
    writes together, some in one column tile and some in two."""
    rs = np.random.default_rng(n + hits)
    shift, rng = 14, 1 << 16
    at = np.arange(n) * 16
    boxes = np.zeros((n, 7), dtype=np.uint32)
    boxes[:, 0], boxes[:, 1] = at, at + 1
    wide = np.arange(0, n, 20)
    first = rs.integers(0, max(1, n - hits), size=len(wide)) * 16
    boxes[wide, 0], boxes[wide, 1] = first, np.minimum(first + 16 * (hits - 1) + 1, (1 << shift) - 1)
    boxes[:, 3] = boxes[:, 5] = 5
    boxes = boxes[rs.permutation(n)]
    boxes[:, 6] = np.arange(n)
    want = O.brute_pairs(boxes)
    red, blue = boxes[:n // 2].copy(), boxes[n // 2:].copy()
    blue[:, 6] = np.arange(len(blue))
    w = want.astype(np.int64)
    w = w[(w[:, 0] < n // 2) & (w[:, 1] >= n // 2)] - [0, n // 2]
    for e in engines:
        for _ in range(2):
            assert e.self_intersect(boxes, rng, cell_shift=shift) == len(want)
        assert np.array_equal(canon(e.pairs()), canon(want))
        for _ in range(2):
            assert e.bipartite_intersect(red, blue, rng, cell_shift=shift) == len(w)
        got = e.pairs().astype(np.int64)
        assert np.array_equal(got[np.lexsort((got[:, 1], got[:, 0]))], w[np.lexsort((w[:, 1], w[:, 0]))])
