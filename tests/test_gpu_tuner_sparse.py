"""Cell sizes of single-scene queries whose usual sizes do not serve: boxes very
small against their spacing, or a few huge boxes among them. Against a
restatement of the device's cost model on the same sampled rows."""
import numpy as np
import pytest

from oracle import oracle as O
from pbig_gb300 import Engine

pytestmark = pytest.mark.gpu
RANGE = 1 << 24


def boxes_of(n, side, seed, dims=3, huge=0):
    r = np.random.default_rng(seed)
    lo = r.integers(0, RANGE - side, size=(n, dims))
    b = np.empty((n, 2 * dims + 1), dtype=np.uint32)
    b[:, 0:2 * dims:2], b[:, 1:2 * dims:2] = lo, lo + side - 1
    for k in range(huge):  # (rows of the sample: every n/4096-th)
        b[(k + 1) * 37 * n >> 12, :2 * dims] = [0, RANGE - 1] * dims
    b[:, -1] = np.arange(n)
    return b


def cells(s, dims):
    return ((RANGE + (1 << s) - 1) >> s) ** dims


def choice(boxes):
    """Costs by size, over the usual sizes and the coarser ones."""
    n, dims = boxes.shape[0], (boxes.shape[1] - 1) // 2
    m = min(n, 4096)
    rows = boxes[[k * n >> 12 for k in range(m)] if n > 4096 else range(m)].astype(np.int64)
    lo, hi = rows[:, 0:2 * dims:2], rows[:, 1:2 * dims:2]
    mean = int((hi - lo + 1).sum()) // (m * dims)
    s0 = mean.bit_length() - 1
    sparse = cells(s0 + 3, dims) > 64 * n
    far = s0 + 3 if sparse else s0 + 5

    def cost(s):
        C = cells(s, dims)
        per = ((hi >> s) - (lo >> s) + 1).prod(axis=1)
        if C > (4000000000 if s <= far else max(4096, 64 * n)) or per.max() >= 1 << 26 or per.sum() > 64 * m:
            return None
        corners = np.unique(lo >> s, axis=0, return_counts=True)[1]
        f = per.sum() / m * (n / m)
        return 3.1e-12 * C + 41e-12 * per.sum() / m * n + 0.46e-12 * int((corners * (corners - 1) // 2).sum()) * f * f

    costs = {s: cost(s) for s in range(max(0, s0 - 2), far + 1)}
    none = all(c is None for c in costs.values())
    if none or (n > 1 << 18 and sparse):
        costs.update({s: cost(s) for s in range(far + 1, 25)})
    return {s: c for s, c in costs.items() if c is not None}, none


@pytest.fixture(scope="module")
def engine():
    e = Engine(0)
    e.set_one_launch(False)
    yield e
    e.close()


@pytest.mark.parametrize("n,side,dims,huge,none", [
    (300000, 2048, 3, 0, False),  # the only usual size makes 2^30 cells
    (300000, 256, 3, 0, True),    # the usual ones make more than there may be
    (262145, 5000, 3, 0, False),
    (262144, 256, 3, 0, True),
    (30000, 16, 3, 0, True),
    (500000, 16, 2, 0, True),
    (400000, 300, 2, 0, False),
    (300000, 500, 3, 1, True),    # the huge box leaves the usual sizes out
])
def test_choice(engine, n, side, dims, huge, none):
    boxes = boxes_of(n, side, n + side, dims, huge)
    costs, without = choice(boxes)
    assert without == none
    engine.self_intersect(boxes, RANGE)
    st = engine.stats()
    shift, best = st["cell_shift"], min(costs.values())
    assert shift in costs and costs[shift] <= best * (1 + 1e-12), (shift, costs)
    assert st["cells"] <= 64 * n and st["grid_retries"] == 0
    want = O.grid_pairs(boxes, RANGE, cs=1 << 18)[0]
    assert np.array_equal(O.sort_pairs(engine.pairs()), want)


@pytest.mark.parametrize("n,side,launches", [
    (20000, 256, 1),      # a coarse grid in the one launch, as self queries have
    (40000, 1200, 1),
    (50000, 100000, 1),   # the usual sizes fit the one launch
])
def test_small_red_blue_queries_run_in_one_launch(n, side, launches):
    both = boxes_of(2 * n, side, n)
    both[n::7, :6] = both[:n][: len(both[n::7]), :6]  # (pairs)
    red, blue = both[:n].copy(), both[n:].copy()
    blue[:, 6] -= n
    p = O.grid_pairs(both, RANGE, cs=1 << 18)[0]
    p = p[(p[:, 0] < n) & (p[:, 1] >= n)]
    with Engine(0) as e:
        assert e.bipartite_intersect(red, blue, RANGE) == len(p) > 2000
        assert e.stats()["kernels"] == launches
        got = e.pairs()
    got[:, 1] += n
    assert np.array_equal(O.sort_pairs(got), p)
