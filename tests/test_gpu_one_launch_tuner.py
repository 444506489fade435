"""The cell size that a one-launch query chooses, against a restatement of its
cost model on the same 64 rows."""
import numpy as np
import pytest

from oracle import oracle as O
from pbig_gb300 import Engine

pytestmark = pytest.mark.gpu
RANGE = 1 << 24


def boxes_of(n, side, dims, seed):
    r = np.random.default_rng(seed)
    lo = r.integers(0, RANGE - side, size=(n, dims))
    b = np.empty((n, 2 * dims + 1), dtype=np.uint32)
    b[:, 0:2 * dims:2], b[:, 1:2 * dims:2] = lo, lo + r.integers(0, side, size=(n, dims))
    b[:, -1] = np.arange(n)
    return b


def choice(b, warps, bip=False):
    n, dims = b.shape[0], (b.shape[1] - 1) // 2
    m = min(n, 64)
    rows = b[[k * n // m for k in range(m)]].astype(np.int64)
    lo, hi = rows[:, 0:2 * dims:2], rows[:, 1:2 * dims:2]
    mean = int((hi - lo + 1).sum()) // (m * dims)
    s0 = mean.bit_length() - 1 if mean >= 2 else 0

    def cost(s, most):
        C = ((RANGE + (1 << s) - 1) >> s) ** dims
        e = int(((hi >> s) - (lo >> s) + 1).prod(axis=1).sum())
        if C > most or e > 64 * m:
            return None
        E = e * (n / m)
        per = (E / C) ** 3
        units = C * max(1, (E / C) ** 2 / 16384)  # a warp's each
        tests = E * E / (2 * C) * max(1, warps / units) * (0.5 if bip else 1)
        return (3e-6 if C > 8192 else 0) + 3.1e-12 * C + 41e-12 * E + 0.5e-9 * C * per / (per + 160) + 2e-12 * tests

    costs = {s: cost(s, 1 << 20) for s in range(max(0, s0 - 2), s0 + 4)}
    if all(c is None for c in costs.values()):  # too sparse in the range for the usual sizes
        costs = {s: cost(s, min(1 << 20, max(4096, 64 * n))) for s in range(s0 + 4, 25)}
    return {s: c for s, c in costs.items() if c is not None}


@pytest.mark.parametrize("dims", [2, 3])
@pytest.mark.parametrize("n,side", [(7000, 300000), (7000, 2), (65536, 100000), (100000, 64), (262144, 64), (262144, 2048),
                                    (200000, 1 << 18)])
def test_choice(dims, n, side):
    import torch
    b = boxes_of(n, side, dims, n + side)
    warps = torch.cuda.get_device_properties(0).multi_processor_count * 16
    with Engine(0) as e:
        count = e.self_intersect(b, RANGE)
        if count * 8 < 1 << 24:
            assert np.array_equal(O.sort_pairs(e.pairs()), O.grid_pairs(b, RANGE, cs=1 << 18)[0])
        e.self_intersect(b, RANGE)  # (a first result too large for the launch's buffers went to the pipeline)
        st = e.stats()
        if st["kernels"] != 1:
            pytest.skip("more pairs or entries than a launch has room for")
        costs = choice(b, warps)
        assert st["cell_shift"] in costs
        # single precision: each term to 1e-6 or better
        assert costs[st["cell_shift"]] <= min(costs.values()) * (1 + 1e-4), (st["cell_shift"], costs)
