"""Single-scene queries where there is no memory for buffers of eight cells and
six entries a box: those of the tuner's estimate fit, and the query runs."""
import numpy as np
import pytest

from oracle import oracle as O
from pbig_gb300 import Engine, PbigError
from pbig_gb300.engine import ENOMEM

pytestmark = pytest.mark.gpu
RANGE = 1 << 24


def scene(n, seed):
    r = np.random.default_rng(seed)
    side = int(0.6 * n ** (-1 / 3) * RANGE)
    lo = r.integers(0, RANGE - side, size=(n, 3))
    b = np.empty((n, 7), dtype=np.uint32)
    b[:, 0:6:2], b[:, 1:6:2] = lo, lo + r.integers(0, side, size=(n, 3))
    b[:, 6] = np.arange(n)
    return b


def canon(p):
    return O.sort_pairs(np.asarray(p, dtype=np.uint32).reshape(-1, 2))


# a query in one launch (its buffers are refused too), and one of several
@pytest.mark.parametrize("n,limit", [(100000, 8 << 20), (300000, 20 << 20)])
@pytest.mark.parametrize("loc", ["host", "device"])
def test_self_queries(n, limit, loc):
    import torch
    boxes = scene(n, n)
    assert 6 * n * 16 > limit  # the entries of a query sized without its estimate
    src = boxes if loc == "host" else torch.from_numpy(boxes.view(np.int32)).cuda()
    with Engine(0) as engine:
        engine.set_max_buffer(limit)
        for _ in range(2):
            assert engine.self_intersect(src, RANGE) == len(O.grid_pairs(boxes, RANGE)[0])
            assert np.array_equal(canon(engine.pairs()), O.grid_pairs(boxes, RANGE)[0])
        engine.set_max_buffer(1 << 20)  # and what does not fit at all is still refused
        with pytest.raises(PbigError) as e:
            engine.self_intersect(scene(2 * n, 1), RANGE)
        assert e.value.code == ENOMEM
        engine.set_max_buffer(0)
        assert engine.self_intersect(src, RANGE) == len(O.grid_pairs(boxes, RANGE)[0])


def test_red_blue_queries():
    n = 150000
    both = scene(2 * n, 7)
    red, blue = both[:n].copy(), both[n:].copy()
    blue[:, 6] -= n
    want = O.grid_pairs(both, RANGE)[0]
    want = want[(want[:, 0] < n) & (want[:, 1] >= n)] - np.array([0, n], dtype=np.uint32)
    with Engine(0) as engine:
        engine.set_max_buffer(20 << 20)
        assert engine.bipartite_intersect(red, blue, RANGE) == len(want)
        assert np.array_equal(canon(engine.pairs()), canon(want))
