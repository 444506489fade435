"""The slots of a resident scene's grid (CPU): their number in 64 bits, against
the sum over the cells, and grids whose slots 32 bits cannot number."""
import numpy as np
import pytest

from pbig_gb300 import engine

LIMIT = (1 << 32) - 1  # starts are 32-bit words, the last of them the number of slots


def slots(ncells, entries):
    return engine.lib().pbig2_scene_slots(ncells, entries)


@pytest.mark.parametrize("ncells,n", [(1, 0), (1, 7), (1000, 1), (1000, 999), (64, 100000)])
def test_no_cells_need_more(ncells, n):
    """A cell of n boxes has n + n/2 + 4 slots."""
    cells = np.random.default_rng(n).integers(0, ncells, size=n)
    count = np.bincount(cells, minlength=ncells)
    need = int((count + count // 2 + 4).sum())
    assert need <= slots(ncells, n) <= need + ncells // 2 + 1


def test_totals_beyond_32_bits_do_not_wrap():
    assert slots(1 << 30, 0) == 1 << 32 > LIMIT          # 2^30 cells: empty ones alone
    assert slots(1 << 27, 1 << 28) < LIMIT               # 2^28 small boxes on their query's grid
    assert slots(1 << 30, 1 << 28) > LIMIT               # and one size finer
    assert slots(1 << 29, 1500000000) == 4 * (1 << 29) + 2250000000 > LIMIT
    assert slots((1 << 30) - 1, 2) == LIMIT + 1 - 4 + 3
    assert slots((1 << 64) - 1, (1 << 64) - 1) == (1 << 64) - 1
