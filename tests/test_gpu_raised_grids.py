"""Automatic cell sizes of a context that has met a box too large for one: every
scene gets the size that its own boxes allow."""
import numpy as np
import pytest

from oracle import oracle as O
from pbig_gb300 import Engine

pytestmark = pytest.mark.gpu
RANGE, N, BIG = 1 << 18, 20001, 12345


def scene(big=None, seed=21):
    """Boxes of side < 64; the tuner's sample has every fifth row, not BIG."""
    r = np.random.default_rng(seed)
    lo = r.integers(0, RANGE - 64, size=(N, 3))
    b = np.empty((N, 7), dtype=np.uint32)
    b[:, 0:6:2], b[:, 1:6:2] = lo, lo + r.integers(0, 64, size=(N, 3))
    b[:, 6] = np.arange(N)
    if big:
        b[BIG, 0:6:2], b[BIG, 1:6:2] = 0, big - 1
    return b


def fits(big, shift):
    return (((big - 1) >> shift) + 1) ** 3 < 1 << 26


def run(e, b):
    n = e.self_intersect(b, RANGE)
    want = O.grid_pairs(b, RANGE, cs=1 << 14)[0]
    assert n == len(want) and np.array_equal(O.sort_pairs(e.pairs()), want)
    st = e.stats()
    return st["cell_shift"], st["grid_retries"]


@pytest.fixture
def engine():
    with Engine(0) as e:
        e.set_one_launch(False)
        yield e


def test_a_plain_scene_keeps_its_own_size(engine):
    plain = run(engine, scene())
    assert plain[1] == 0 and not fits(RANGE, plain[0])
    raised, retries = run(engine, scene(RANGE))
    assert retries == raised - plain[0] > 0 and fits(RANGE, raised) and not fits(RANGE, raised - 1)
    assert run(engine, scene()) == plain
    assert run(engine, scene(RANGE)) == (raised, 0)
    assert run(engine, scene(seed=22))[0] == plain[0]


def test_each_scene_is_raised_as_far_as_it_needs(engine):
    plain = run(engine, scene())[0]
    most = run(engine, scene(RANGE))[0]
    for big in (RANGE // 2, RANGE, 1000, RANGE // 2 + 77):
        shift, retries = run(engine, scene(big))
        assert retries == 0 and fits(big, shift) and (shift == plain or not fits(big, shift - 1)), big
        assert plain <= shift <= most


def test_red_blue_and_self_queries_apart(engine):
    """(of one number of boxes)"""
    b = scene(RANGE)
    run(engine, b)
    red, blue = scene()[:10000].copy(), scene()[10000:].copy()
    blue[:, 6] -= 10000
    engine.bipartite_intersect(red, blue, RANGE)
    st = engine.stats()
    assert not fits(RANGE, st["cell_shift"]) and st["grid_retries"] == 0
