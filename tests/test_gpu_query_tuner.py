"""The cell size a single-scene query chooses on the device, against a
restatement of its cost model on the same sampled rows, and that the choice
does not depend on the queries before it."""
import numpy as np
import pytest

from oracle import oracle as O
from pbig_gb300 import Engine, gen

pytestmark = pytest.mark.gpu


def choice(boxes, rng, bip=False):
    """The device tuner restated: costs of every size it may take, by size."""
    n, dims = boxes.shape[0], (boxes.shape[1] - 1) // 2
    m = min(n, 4096)
    rows = boxes[[k * n >> 12 for k in range(m)] if n > 4096 else range(m)].astype(np.int64)
    lo, hi = rows[:, 0:2 * dims:2], rows[:, 1:2 * dims:2]
    ok = ((lo <= hi) & (hi < rng)).all(axis=1)
    lo, hi = lo[ok], hi[ok]
    mean = int((hi - lo + 1).sum()) // (max(1, len(lo)) * dims)
    s0 = mean.bit_length() - 1 if mean >= 2 else 0
    win = min(31, s0 + 3)
    far = min(31, s0 + 5) if ((rng + (1 << win) - 1) >> win) ** dims <= 64 * n else win
    costs = {}
    for s in range(max(0, s0 - 2), far + 1):
        C = ((rng + (1 << s) - 1) >> s) ** dims
        cells = ((hi >> s) - (lo >> s) + 1).prod(axis=1)
        if C > 4000000000 or cells.max() >= 1 << 26 or cells.sum() > 64 * m:
            continue
        corners = np.unique(lo >> s, axis=0, return_counts=True)[1]
        pairs = int((corners * (corners - 1) // 2).sum())
        per_box = cells.sum() / m
        f = per_box * (n / m)
        costs[s] = 3.1e-12 * C + 41e-12 * per_box * n + (0.5 if bip else 1.0) * 0.46e-12 * pairs * f * f
    return costs


def check(shift, costs):
    best = min(costs.values())
    assert shift in costs and costs[shift] <= best * (1 + 1e-12), (shift, costs)  # (the sums round apart by less)


SCENES = {
    "clustered": lambda: (gen.clustered3d(300007, seed=3), gen.RANGE),
    "plain2d": lambda: (gen.uniform2d(50001, seed=4), gen.RANGE),
    "scene of 4096": lambda: (gen.scene3d(4096, 5), gen.RANGE),
    "scene of 4097": lambda: (gen.scene3d(4097, 6), gen.RANGE),
    "two sizes": lambda: (gen.mixed3d(100003, seed=7), gen.RANGE),
    "crowded": lambda: (O.harness_boxes(200000, sim="UN"), 10000),
    "three boxes": lambda: (gen.scene3d(3, 8), gen.RANGE),
}


@pytest.fixture(scope="module")
def engine():
    e = Engine(0)
    e.set_one_launch(False)
    yield e
    e.close()


@pytest.mark.parametrize("where", ["device", "pageable", "page-locked", "device, odd rows"])
@pytest.mark.parametrize("name", SCENES)
def test_choice_of_a_self_query(engine, name, where):
    import torch
    boxes, rng = SCENES[name]()
    costs = choice(boxes, rng)
    src = torch.from_numpy(boxes.view(np.int32))
    if where == "device":
        src = src.cuda()
    elif where == "page-locked":
        src = src.pin_memory()
    elif where == "pageable":
        src = boxes
    else:  # rows that begin at every multiple of 4 bytes
        room = torch.zeros(boxes.size + 3, dtype=torch.int32, device="cuda")
        src = room[3:3 + boxes.size].view(boxes.shape)
        src.copy_(torch.from_numpy(boxes.view(np.int32)))
    engine.self_intersect(src, rng)
    check(engine.stats()["cell_shift"], costs)


def test_choice_of_red_and_blue(engine):
    red, blue = gen.mixed3d(70001, seed=9), gen.mixed3d(30002, seed=10)
    engine.bipartite_intersect(red, blue, gen.RANGE)
    check(engine.stats()["cell_shift"], choice(np.concatenate([red, blue]), gen.RANGE, bip=True))


def test_choice_is_the_scenes_own(engine):
    """Two scenes of one size and one mean extent, one crowded: each keeps its
    own cell size whichever came first."""
    n = 100000
    even = gen.scene3d(n, 11)
    crowded = even.copy()
    crowded[:, :6] = (even[:, :6] // 16) + gen.RANGE // 3
    side = (even[:, 1:6:2] - even[:, 0:6:2])
    crowded[:, 1:6:2] = np.minimum(crowded[:, 0:6:2] + side, gen.RANGE - 1)
    for boxes in (even, crowded, even):
        engine.self_intersect(boxes, gen.RANGE)
        check(engine.stats()["cell_shift"], choice(boxes, gen.RANGE))
