"""Batched results grouped by scene: from two scenes to more than the grouping
counts in shared memory, empty scenes among them, against each scene's own
brute force, and a smaller batch after a larger one (the captured pipeline of
the larger serves it)."""
import numpy as np
import pytest

from oracle import oracle as O
from pbig_gb300 import Engine, gen

pytestmark = pytest.mark.gpu


def batch(sizes, seed):
    parts = [gen.scene3d(int(n), seed + i) if n else np.empty((0, 7), np.uint32) for i, n in enumerate(sizes)]
    return np.concatenate(parts), np.concatenate([[0], np.cumsum(sizes)]).astype(np.uint64), parts


def check(e, boxes, offs, parts, src):
    total = e.batch_intersect(src, offs, gen.RANGE)
    so = e.scene_offsets().astype(np.int64)
    got = e.pairs().astype(np.int64)
    assert so[0] == 0 and so[-1] == total == len(got)
    for i, part in enumerate(parts):
        mine = got[so[i]:so[i + 1]]
        if len(part) < 2:
            assert len(mine) == 0, i
            continue
        want = O.brute_pairs(part)
        assert np.array_equal(mine[np.lexsort((mine[:, 1], mine[:, 0]))], want), i


@pytest.mark.parametrize("sizes", [[1000, 3], [0, 5000, 0, 4096, 1, 257], [64] * 33, [7] * 1025], ids=lambda s: f"{len(s)} scenes")
def test_few_and_many_scenes(sizes):
    boxes, offs, parts = batch(sizes, 100)
    with Engine(0) as e:
        check(e, boxes, offs, parts, boxes)


def test_more_scenes_than_shared_counters():
    rs = np.random.default_rng(5)
    boxes, offs, parts = batch(rs.integers(0, 12, size=12290), 1000)
    import torch
    dev = torch.from_numpy(boxes.view(np.int32)).cuda()
    with Engine(0) as e:
        for n in (12290, 8193, 8192, 50):  # the later ones may run the pipeline captured for the first
            check(e, boxes, offs[:n + 1], parts[:n], dev[:int(offs[n])])
