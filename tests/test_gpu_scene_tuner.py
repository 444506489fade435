"""The per-scene cell sizes of batches against a model of the tuner in Python
(the same rows, integers and double-precision operations): scenes of one box to
thousands, 2-D and 3-D, boxes of a point to the whole range, invalid boxes, and
scenes for which no size of the window qualifies. Exactly equal."""
import numpy as np
import pytest

from pbig_gb300 import Engine, PbigError
from pbig_gb300.engine import EINPUT

pytestmark = pytest.mark.gpu


def model(rows, dims, rng):
    n = len(rows)
    m = min(n, 64)
    nrc = lambda s: (rng + (1 << s) - 1) >> s
    single = next(s for s in range(32) if nrc(s) <= 1 or s == 31)
    if m == 0:
        return single
    r = rows[(np.arange(m) * n) // m].astype(object)
    lo, hi = r[:, 0:2 * dims:2], r[:, 1:2 * dims:2]
    ok = np.array([all(a <= b < rng for a, b in zip(x, y)) for x, y in zip(lo, hi)])
    lo, hi = lo[ok], hi[ok]
    mean = float(sum(int(b) - int(a) + 1 for x, y in zip(lo, hi) for a, b in zip(x, y))) / float(max(1, len(lo)) * dims)
    s0 = int(mean).bit_length() - 1 if mean >= 2.0 else 0
    win = min(s0 + 3, 31)

    def cost(s, far):
        C = float(nrc(s))
        for _ in range(1, dims):
            C = C * float(nrc(s))
        cells = []
        for x, y in zip(lo, hi):
            c = 1
            for a, b in zip(x, y):
                c *= (int(b) >> s) - (int(a) >> s) + 1
            cells.append(c)
        e = sum(cells)
        if C > 4.0e9 or (far and C > max(4096.0, 64.0 * n)) or any(c >= 1 << 26 for c in cells) or e > 64 * m:
            return None
        E = float(e) * (float(n) / float(m))
        T = E * E / (2.0 * C)
        occ = 2.0 * T / (E if E > 1.0 else 1.0) + 1.0
        f = occ / 96.0 if occ / 96.0 > 1.0 else 1.0
        return 2.4e-12 * C + 80.0e-12 * E + 0.9e-12 * f * T

    for sizes, far in ((range(max(0, s0 - 2), win + 1), False), (range(win + 1, 32), True)):
        found = [(c, s) for s in sizes if (c := cost(s, far)) is not None]
        if found:
            return min(found)[1]
    return single


@pytest.mark.parametrize("dims", [2, 3])
@pytest.mark.parametrize("rng", [2, 1000, 1 << 20, 1 << 24, (1 << 32) - 1])
def test_every_scene_gets_the_models_size(dims, rng):
    rs = np.random.default_rng(dims * 1000 + rng % 997)
    scenes = []
    for n in (1, 2, 31, 63, 64, 65, 100, 1000, 5000):
        for side in (1, max(1, rng // 5000), max(1, rng // 100), rng):
            if n > 100 and side > rng // 100 and rng > 1000:
                continue  # (everything overlaps)
            lo = rs.integers(0, rng, size=(n, dims), dtype=np.int64)
            hi = np.minimum(lo + rs.integers(0, side, size=(n, dims)), rng - 1)
            b = np.empty((n, 2 * dims + 1), dtype=np.uint32)
            b[:, 0:2 * dims:2], b[:, 1:2 * dims:2], b[:, -1] = lo, hi, np.arange(n)
            if n == 100:  # invalid rows among the sampled ones
                b[0, 0], b[0, 1] = 1, 0
            if n == 1000:  # a sampled box that spans the range
                b[0, 0:2 * dims:2], b[0, 1:2 * dims:2] = 0, rng - 1
            scenes.append(b if rng > 1000 or n <= 100 else b[:64])
    offs = np.concatenate([[0], np.cumsum([len(b) for b in scenes])])
    with Engine(0) as e:
        try:
            e.batch_intersect(np.concatenate(scenes), offs, rng)
        except PbigError as err:  # (the invalid rows are skipped and reported)
            assert err.code == EINPUT
        assert e.stats()["grid_retries"] == 0
        assert list(e.scene_shifts(len(scenes))) == [model(b, dims, rng) for b in scenes]
