"""Cells whose boxes overlap nearly all of one another: tile steps with more
pairs than a warp's buffer holds, and cells with many tile tasks."""
import numpy as np
import pytest

from oracle import oracle as O
from pbig_gb300 import Engine

pytestmark = pytest.mark.gpu
RANGE = 1 << 20


@pytest.fixture(scope="module")
def engines():
    one, many = Engine(0), Engine(0)
    many.set_one_launch(False)
    yield one, many
    one.close()
    many.close()


def dense(n, dims, share, seed):
    """n boxes that fill `share` of the range along every axis."""
    r = np.random.default_rng(seed)
    side = int(share * RANGE)
    lo = r.integers(0, RANGE - side, size=(n, dims))
    b = np.empty((n, 2 * dims + 1), dtype=np.uint32)
    b[:, 0:2 * dims:2], b[:, 1:2 * dims:2] = lo, lo + side
    b[:, -1] = np.arange(n)
    return b


def canon(p):
    return O.sort_pairs(np.asarray(p, dtype=np.uint32).reshape(-1, 2))


@pytest.mark.parametrize("dims", [2, 3])
@pytest.mark.parametrize("share", [0.9, 0.45])
@pytest.mark.parametrize("n", [33, 64, 127, 129, 511, 513, 545, 1030, 6145])
def test_self_queries(engines, dims, share, n):
    """In one cell, then at the size that the query chooses; a first result too
    large for the pair buffer is redone."""
    boxes = dense(n, dims, share, n + dims)
    want = O.brute_pairs(boxes)
    for e in engines:
        for shift in (20, 20, None, None):
            assert e.self_intersect(boxes, RANGE, cell_shift=shift) == len(want), shift
        assert np.array_equal(canon(e.pairs()), want)


@pytest.mark.parametrize("red,blue", [(33, 31), (64, 64), (400, 100), (513, 600), (4000, 3000)])
def test_red_blue_queries(engines, red, blue):
    both = dense(red + blue, 3, 0.6, red)
    want = O.brute_pairs(both)
    want = want[(want[:, 0] < red) & (want[:, 1] >= red)] - np.array([0, red], dtype=np.uint32)
    b = both[red:].copy()
    b[:, -1] -= np.uint32(red)
    for e in engines:
        for shift in (20, 20, None):
            assert e.bipartite_intersect(both[:red].copy(), b, RANGE, cell_shift=shift) == len(want), shift
        got = e.pairs()
        assert np.array_equal(got[np.lexsort((got[:, 1], got[:, 0]))], want)


def test_pairs_beyond_the_callers_buffer(engines):
    """The count is right and nothing is written past the end."""
    import torch
    boxes = dense(1500, 3, 0.9, 3)
    want = O.brute_pairs(boxes)
    room = torch.full((len(want) // 2 + 64, 2), -1, dtype=torch.int32, device="cuda")
    for e in engines:
        e.set_pair_output(room[: len(want) // 2])
        assert e.self_intersect(boxes, RANGE, cell_shift=20) == len(want)
        assert not e.result_in(room[: len(want) // 2]) and np.array_equal(canon(e.pairs()), want)
        assert bool((room[len(want) // 2:] == -1).all())
        e.set_pair_output(None)


def test_a_query_of_many_tile_tasks_runs_in_one_launch_again():
    """A launch short of room for its tile tasks goes to the pipeline once."""
    boxes = dense(12000, 2, 0.3, 5)
    with Engine(0) as e:
        e.self_intersect(boxes, RANGE, cell_shift=19)
        count = e.self_intersect(boxes, RANGE, cell_shift=19)
        assert e.stats()["kernels"] == 1 and count == len(O.grid_pairs(boxes, RANGE, cs=1 << 19)[0])
