"""Statistics of a query do not depend on how it was launched."""
import numpy as np
import pytest

from pbig_gb300 import Engine

pytestmark = pytest.mark.gpu
RANGE = 1 << 20


def boxes_of(n, seed):
    r = np.random.default_rng(seed)
    lo = r.integers(0, RANGE - 5000, size=(n, 3))
    b = np.empty((n, 7), dtype=np.uint32)
    b[:, 0:6:2], b[:, 1:6:2] = lo, lo + r.integers(0, 5000, size=(n, 3))
    b[:, 6] = np.arange(n)
    return b


@pytest.mark.parametrize("n", [50, 3000, 20000])
@pytest.mark.parametrize("one_launch", [True, False])
def test_scenes_and_boxes(n, one_launch):
    """A red/blue query has two scenes, a self query one."""
    red, blue = boxes_of(n, 1), boxes_of(n + 7, 2)
    with Engine(0) as e:
        e.set_one_launch(one_launch)
        for _ in range(2):
            e.bipartite_intersect(red, blue, RANGE)
            st = e.stats()
            assert (st["scenes"], st["boxes"]) == (2, 2 * n + 7)
            e.self_intersect(red, RANGE)
            st = e.stats()
            assert (st["scenes"], st["boxes"]) == (1, n)


def test_phases_of_pair_kernels_beside_each_other():
    """Pairs bound for page-locked memory: one time for the three pair kernels,
    none of their own; alone they have theirs."""
    import torch
    boxes = boxes_of(300000, 3)
    host = torch.empty(4000000, 2, dtype=torch.int32).pin_memory()
    names = ("pairs_small", "pairs_med", "pairs_block")
    with Engine(0) as e:
        e.set_pair_output(host)
        e.self_intersect(boxes, RANGE)
        ph = e.stats()["phase_ms"]
        assert e.result_in(host) and ph["pairs"] > 0 and [ph[k] for k in names] == [0, 0, 0]
        e.set_host_split(-1)
        e.self_intersect(boxes, RANGE)
        ph = e.stats()["phase_ms"]
        assert all(ph[k] > 0 for k in names) and abs(sum(ph[k] for k in names) - ph["pairs"]) < 1e-6
        e.set_pair_output(None)
        e.self_intersect(boxes, RANGE)
        assert all(e.stats()["phase_ms"][k] > 0 for k in names)
