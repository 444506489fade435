"""Queries small enough to test every pair of tiles: sizes around the tiles and
the limit of the rule, both dimensions, ranges up to 2^31 (a wider one has no
grid of one cell and takes the grid), invalid boxes, red and blue boxes, and
that the path is not taken where a grid was asked for."""
import numpy as np
import pytest

from oracle import oracle as O
from pbig_gb300 import Engine, gen
from pbig_gb300.engine import EINPUT

pytestmark = pytest.mark.gpu
LIMIT = 6144


@pytest.fixture(scope="module")
def engine():
    e = Engine(0)
    yield e
    e.close()


def scene(n, dims, rng, seed):
    rs = np.random.default_rng(seed)
    side = max(2, int(rng * (1.5 / max(n, 2)) ** (1 / dims)))
    lo = rs.integers(0, rng, size=(n, dims), dtype=np.int64)
    hi = np.minimum(lo + rs.integers(0, min(side, rng), size=(n, dims)), rng - 1)
    rows = np.empty((n, 2 * dims + 1), dtype=np.uint32)
    rows[:, 0:2 * dims:2], rows[:, 1:2 * dims:2], rows[:, -1] = lo, hi, np.arange(n)
    return rows


def canon(p):
    return O.sort_pairs(np.asarray(p, dtype=np.uint32).reshape(-1, 2))


def cross(red, blue):
    u = np.concatenate([red, blue])
    u[:, -1] = np.arange(len(u))
    p = O.brute_pairs(u).astype(np.int64)
    p = p[(p[:, 0] < len(red)) & (p[:, 1] >= len(red))]
    p[:, 1] -= len(red)
    return p


@pytest.mark.parametrize("dims", [2, 3])
@pytest.mark.parametrize("rng", [1, 2, 1000, 1 << 24, 1 << 31, (1 << 31) + 1, (1 << 32) - 1])
def test_self_queries(engine, dims, rng):
    for n in (1, 2, 31, 32, 33, 64, 65, 1000, LIMIT, LIMIT + 1):
        if rng < 1000 and n > 100:
            continue  # (everything overlaps)
        boxes = scene(n, dims, rng, n + dims)
        want = O.brute_pairs(boxes)
        for _ in range(2):  # (a first result too large for the buffer is redone)
            assert engine.self_intersect(boxes, rng) == len(want), n
            assert np.array_equal(canon(engine.pairs()), want), n
        st = engine.stats()
        if n <= LIMIT and rng <= 1 << 31:
            assert st["kernels"] == 1 and st["cells"] == 1 and 1 << st["cell_shift"] >= rng
            assert st["entries"] == n and st["pair_tests"] == n * (n - 1) // 2


@pytest.mark.parametrize("dims", [2, 3])
def test_red_and_blue(engine, dims):
    import torch
    for nr, nb in [(0, 5), (5, 0), (1, 1), (32, 33), (1, 700), (700, 31), (3000, 3144), (3000, 3145)]:
        red, blue = scene(nr, dims, 1 << 20, 7 * nr + dims), scene(nb, dims, 1 << 20, 5 * nb + 100)
        want = cross(red, blue)
        for place in ("host", "device"):
            a, b = (torch.from_numpy(v.view(np.int32)).cuda() if place == "device" else v for v in (red, blue))
            for _ in range(2):
                assert engine.bipartite_intersect(a, b, 1 << 20) == len(want), (nr, nb, place)
            got = engine.pairs().astype(np.int64)
            assert np.array_equal(got[np.lexsort((got[:, 1], got[:, 0]))], want), (nr, nb, place)


@pytest.mark.parametrize("n", [40, 5000])
def test_invalid_boxes_are_skipped_and_counted(engine, n):
    rng = 1 << 16
    boxes = scene(n, 3, rng, 3)
    bad = [0, 33, n - 1]
    boxes[0, 1] = rng            # a coordinate beyond the range
    boxes[33, 2:4] = [9, 3]      # inverted
    boxes[n - 1, 6] = 0          # another box's index
    good = np.delete(boxes, bad, axis=0)
    keep = np.delete(np.arange(n), bad)
    good[:, 6] = np.arange(len(good))
    want = keep[O.brute_pairs(good).astype(np.int64)]
    assert engine.self_intersect(boxes, rng, allow_bad=True) == len(want)
    assert engine.last_rc == EINPUT and engine.stats()["bad_boxes"] == 3
    assert np.array_equal(canon(engine.pairs()), canon(want))


def test_bad_boxes_of_a_colour_alone(engine):
    from pbig_gb300 import PbigError
    red = scene(50, 3, 1 << 16, 4)
    red[7, 0] = 1 << 16
    for a, b in ((red, red[:0]), (red[:0], red)):
        with pytest.raises(PbigError) as e:
            engine.bipartite_intersect(a, b, 1 << 16)
        assert e.value.code == EINPUT and engine.stats()["bad_boxes"] == 1


def test_a_grid_where_it_was_asked_for(engine):
    boxes = gen.scene3d(2000, 5)
    want = O.brute_pairs(boxes)
    for shift in (21, 24):
        assert engine.self_intersect(boxes, gen.RANGE, cell_shift=shift) == len(want)
        assert engine.stats()["cell_shift"] == shift
    engine.set_class_map(0x6666665544321000)
    try:
        assert engine.self_intersect(boxes, gen.RANGE) == len(want)
        assert engine.stats()["cells"] > 1
    finally:
        engine.set_class_map(0)
    # a resident scene's grid
    from pbig_gb300 import Scene
    sc = Scene(engine, boxes, gen.RANGE)
    assert sc.npairs == len(want) and engine.stats()["cells"] > 1
    sc.close()


@pytest.mark.parametrize("n", [6200, 20000, 131072])
def test_red_and_blue_in_one_launch(engine, n):
    """Red and blue boxes between the all-pairs rule and the one-launch limit,
    colours of very different counts, device arrays of their own."""
    import torch
    for nr in (n // 2, 3, n - 33):
        red, blue = gen.mixed3d(nr, seed=n + nr), gen.mixed3d(n - nr, seed=n + nr + 1)
        want = cross(red, blue)
        a, b = (torch.from_numpy(v.view(np.int32)).cuda() for v in (red, blue))
        for _ in range(2):
            assert engine.bipartite_intersect(a, b, gen.RANGE) == len(want), nr
        assert engine.stats()["kernels"] == 1
        got = engine.pairs().astype(np.int64)
        assert np.array_equal(got[np.lexsort((got[:, 1], got[:, 0]))], want), nr


def uneven(n, dims, rng, seed):
    """Small boxes, and one in 700 that covers a third of the range along one axis
    (hundreds of cells, all of one warp's boxes small but one)."""
    rs = np.random.default_rng(seed)
    rows = scene(n, dims, rng, seed)
    for k in rs.choice(n, max(1, n // 700), replace=False):
        a = int(rs.integers(0, dims))
        rows[k, 2 * a] = rs.integers(0, rng // 2)
        rows[k, 2 * a + 1] = rows[k, 2 * a] + rng // 3
    return rows


@pytest.mark.parametrize("dims", [2, 3])
@pytest.mark.parametrize("n", [6145, 77824, 77825, 100000, 262144])
def test_boxes_of_very_different_cell_counts_in_one_launch(engine, n, dims):
    """Parts of the boxes below, at and above a block's tile of 512 on 152 SMs."""
    rng = 1 << 24
    boxes = uneven(n, dims, rng, n + dims)
    red, blue = boxes[:n // 3].copy(), boxes[n // 3:].copy()
    red[:, -1], blue[:, -1] = np.arange(len(red)), np.arange(len(blue))
    want = O.grid_pairs(boxes, rng)[0] if n > 20000 else O.brute_pairs(boxes)
    w = want.astype(np.int64)
    w = w[(w[:, 0] < len(red)) & (w[:, 1] >= len(red))] - [0, len(red)]
    for _ in range(2):
        assert engine.self_intersect(boxes, rng) == len(want)
    assert engine.stats()["kernels"] == 1
    assert np.array_equal(canon(engine.pairs()), canon(want))
    for _ in range(2):
        assert engine.bipartite_intersect(red, blue, rng) == len(w)
    assert engine.stats()["kernels"] == 1
    got = engine.pairs().astype(np.int64)
    assert np.array_equal(got[np.lexsort((got[:, 1], got[:, 0]))], w[np.lexsort((w[:, 1], w[:, 0]))])
