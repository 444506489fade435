"""The queries this engine is measured on: what they are, their inputs, and one pass through each.

The kinds of scene are those of the package's generators and of the reference's harness, drawn
here on the GPU so that inputs are quick to make: `scene` (uniform centres, sides in proportion to
n^(-1/3): the batched and serving scenes), `plain2d` (the plain 2-D scene), `clustered` (64
Gaussians, lognormal sides), `redblue` (uniform, 1 % large boxes, only red-blue pairs), `harness`
(integer coordinates below 10 000, sides below 100, positions uniform or normal). A program keeps
one Engine and gives every query's pairs a buffer of its own, as these cases do.

Pairs are whole numbers, so a result is right or wrong and there is no `exact`.
"""
import math

import numpy as np
import torch

from pbig_gb300 import Engine, Scene

RANGE = 1 << 24            # the generators' coordinate range
WIDE = (1 << 32) - 1       # boxes quantised to the whole 32-bit range
HARNESS = 10000            # the reference harness's range; its sides are below 100

_engine = None


def engine():
    global _engine
    if _engine is None:
        _engine = Engine(0)
    return _engine


def listed():
    return [
        # the smallest request of the serving loop: latency
        {"name": "scene 1k", "kind": "scene", "n": 1024, "range": RANGE},
        # a mid-sized request
        {"name": "scene 30k", "kind": "scene", "n": 30011, "range": RANGE},
        # the plain 2-D self-intersection
        {"name": "plain2d 64k", "kind": "plain2d", "n": 65536, "range": RANGE},
        # a large request, odd size
        {"name": "scene 500k", "kind": "scene", "n": 500009, "range": RANGE},
        # the headline scene: skewed cell occupancy, about 9 overlaps per box
        {"name": "clustered 4M", "kind": "clustered", "n": 4194304, "range": RANGE},
        # the same distribution in coordinates that use all 32 bits
        {"name": "clustered 1M wide", "kind": "clustered", "n": 1000003, "range": WIDE},
        # red/blue queries: a small one and the headline size
        {"name": "redblue 25k", "kind": "redblue", "n": 20011, "n_blue": 30013, "range": RANGE},
        {"name": "redblue 2M", "kind": "redblue", "n": 2097152, "n_blue": 2097152, "range": RANGE},
        # the reference benchmark's crowded scene: about 45 overlaps per box, cells of hundreds of boxes
        {"name": "harness normal 4M", "kind": "harness", "n": 4000000, "normal": True, "range": HARNESS},
        # independent scenes in one call: a large batch, and what the serving loop admits at once
        {"name": "batch 512", "kind": "batch", "scenes": 512, "lo": 256, "hi": 262144, "range": RANGE},
        {"name": "batch 8", "kind": "batch", "scenes": 8, "lo": 1024, "hi": 1048576, "range": RANGE},
        # a resident scene of which 1 % of the boxes move
        {"name": "update 1M", "kind": "update", "n": 1048576, "moved": 10485, "range": RANGE},
    ]


def _spread(rng, lo, hi):
    """An integer between lo and hi, even over the logarithm."""
    return max(lo, min(hi, int(math.exp(rng.uniform(math.log(lo), math.log(hi))))))


def draw(rng):
    kind = rng.choice(["scene", "plain2d", "clustered", "redblue", "harness", "batch", "update"])
    if kind == "scene":
        return {"kind": kind, "n": _spread(rng, 1024, 1048576), "range": RANGE}
    if kind == "plain2d":
        return {"kind": kind, "n": _spread(rng, 4096, 1048576), "range": RANGE}
    if kind == "clustered":
        return {"kind": kind, "n": _spread(rng, 65536, 4194304), "range": rng.choice([RANGE, RANGE, WIDE])}
    if kind == "redblue":
        return {"kind": kind, "n": _spread(rng, 16384, 2097152), "n_blue": _spread(rng, 16384, 2097152), "range": RANGE}
    if kind == "harness":
        return {"kind": kind, "n": _spread(rng, 131072, 4000000), "normal": rng.random() < 0.5, "range": HARNESS}
    if kind == "batch":
        scenes = _spread(rng, 4, 512)
        return {"kind": kind, "scenes": scenes, "lo": 256, "hi": 1048576 if scenes <= 16 else 262144, "range": RANGE}
    n = _spread(rng, 65536, 1048576)
    return {"kind": kind, "n": n, "moved": max(1, n // 100), "range": RANGE}


# ---- inputs -----------------------------------------------------------------

def _random(seed):
    return torch.Generator(device="cuda").manual_seed(seed)


def _uniform(gen, n, dims, lo, hi):
    return lo + (hi - lo) * torch.rand(n, dims, generator=gen, device="cuda", dtype=torch.float64)


def _rows(low, high, limit):
    """RectInfo rows of boxes in [0, 1): [min, max] per axis, then the index within the scene."""
    n, dims = low.shape
    rows = torch.empty(n, 2 * dims + 1, dtype=torch.int64, device="cuda")
    rows[:, 0:2 * dims:2] = (low * limit).floor_().clamp_(0, limit - 1)
    rows[:, 1:2 * dims:2] = (high * limit).floor_().clamp_(0, limit - 1)
    rows[:, 2 * dims] = torch.arange(n, device="cuda")
    return rows.to(torch.int32)  # the bits of the unsigned coordinates


def _scene(gen, n, limit):
    half = 0.25 * n ** (-1.0 / 3.0) * _uniform(gen, n, 3, 0.5, 2.0)
    centre = _uniform(gen, n, 3, 0.0, 1.0)
    return _rows(centre - half, centre + half, limit)


def _boxes(case, gen):
    kind, n, limit = case["kind"], case["n"], case["range"]
    if kind == "plain2d":
        low = _uniform(gen, n, 2, 0.0, 1.0)
        return _rows(low, low + _uniform(gen, n, 2, 0.001, 0.005), limit)
    if kind == "clustered":
        means = _uniform(gen, 64, 3, 0.1, 0.9)
        centre = means[torch.randint(64, (n,), generator=gen, device="cuda")]
        centre = (centre + 0.02 * torch.randn(n, 3, generator=gen, device="cuda", dtype=torch.float64)).clamp_(0, 1)
        half = 0.001 * torch.exp(0.5 * torch.randn(n, 3, generator=gen, device="cuda", dtype=torch.float64))
        return _rows(centre - half, centre + half, limit)
    if kind == "harness":
        if case["normal"]:
            low = limit / 2 + limit / 10 * torch.randn(n, 3, generator=gen, device="cuda", dtype=torch.float64)
        else:
            low = _uniform(gen, n, 3, 0, limit)
        low = low.floor_().clamp_(0, limit - 1)
        side = torch.randint(100, (n, 3), generator=gen, device="cuda")
        return _rows((low + 0.5) / limit, (low + side + 0.5) / limit, limit)
    return _scene(gen, n, limit)


def _mixed(gen, n, limit):
    small = _uniform(gen, n, 3, 0.001, 0.004)
    large = _uniform(gen, n, 3, 0.02, 0.1)
    is_large = torch.rand(n, 1, generator=gen, device="cuda") < 0.01
    half = 0.5 * torch.where(is_large, large, small)
    centre = _uniform(gen, n, 3, 0.0, 1.0)
    return _rows(centre - half, centre + half, limit)


def _sizes(case):
    """The scene sizes of a batch: even over the logarithm, the same set for every seed."""
    m, lo, hi = case["scenes"], case["lo"], case["hi"]
    return [int(lo * (hi / lo) ** ((i * 0.6180339887498949) % 1.0)) for i in range(1, m + 1)]


def _moved(case, gen, rows):
    """Indices of the boxes that move, and their rows after a step of N(0, 0.001) per axis."""
    k, limit = case["moved"], case["range"]
    idx = torch.randperm(case["n"], generator=gen, device="cuda")[:k].sort().values
    step = 0.001 * limit * torch.randn(k, 3, generator=gen, device="cuda", dtype=torch.float64)
    old = rows[idx].to(torch.int64)
    new = old.clone()
    for d in range(3):
        by = step[:, d].round().to(torch.int64)
        new[:, 2 * d] = (old[:, 2 * d] + by).clamp_(0, limit - 1)
        new[:, 2 * d + 1] = (old[:, 2 * d + 1] + by).clamp_(0, limit - 1)
    return idx, old, new


def _pairs_of(case):
    """About how many pairs a case has."""
    kind = case["kind"]
    if kind == "batch":
        return 0.98 * sum(_sizes(case))
    n = case["n"]
    if kind == "plain2d":
        return 0.5 * n * n * 0.006 ** 2
    if kind == "clustered":
        return 2.1e-6 * n * n
    if kind == "harness":
        return (1.12e-5 if case["normal"] else 5.0e-7) * n * n
    if kind == "redblue":
        return 5.1e-6 * n * case["n_blue"]
    return 0.98 * n


def _page_locked(t):
    """A page-locked host array with t's rows, as the engine takes them."""
    return t.to(torch.int32).cpu().pin_memory().numpy().view(np.uint32)


def prepare(case, seed):
    gen = _random(seed)
    state = {"kind": case["kind"], "range": case["range"]}
    if case["kind"] == "update":
        rows = _boxes(case, gen)
        idx, old, new = _moved(case, gen, rows)
        engine().set_pair_output(None)
        state["scene"] = Scene(engine(), rows, case["range"])
        state["idx"] = _page_locked(idx)
        state["next"], state["after"] = _page_locked(new), _page_locked(old)
        state["room"] = int(1.5 * _pairs_of(case))
        changed = torch.zeros(16 * case["moved"] + 4096, 2, device="cuda")
        state["removed"], state["added"] = _page_locked(changed), _page_locked(changed)
        return state
    if case["kind"] == "batch":
        sizes = _sizes(case)
        state["boxes"] = torch.cat([_scene(gen, n, case["range"]) for n in sizes])
        state["offsets"] = np.concatenate([[0], np.cumsum(sizes)]).astype(np.uint64)
    elif case["kind"] == "redblue":
        state["boxes"] = _mixed(gen, case["n"], case["range"])
        state["blue"] = _mixed(gen, case["n_blue"], case["range"])
    else:
        state["boxes"] = _boxes(case, gen)
    state["out"] = torch.empty(int(1.5 * _pairs_of(case)) + 16384, 2, dtype=torch.int32, device="cuda")
    return state


# ---- a pass -----------------------------------------------------------------

class Found(dict):
    """A query's result by name. The engine reports pairs in no particular order, as the
    reference does, so a list of pairs comes out of here sorted, to be compared with another,
    and filled up with -1 to the room its caller had for it."""

    def __init__(self, room, **found):
        super().__init__(found)
        self.room = room

    def __getitem__(self, name):
        found = super().__getitem__(name)
        if isinstance(found, Scene):
            found = found.pairs()
        if isinstance(found, np.ndarray) and found.ndim == 2:
            found = torch.from_numpy(found.view(np.int32)).cuda()
        if not isinstance(found, torch.Tensor):
            return found
        first, second = found[:, 0].to(torch.int64), found[:, 1].to(torch.int64)
        if "offsets" in self:  # pairs of many scenes, grouped: sorted within each
            many = np.diff(super().__getitem__("offsets").astype(np.int64))
            scene = torch.from_numpy(np.repeat(np.arange(len(many)), many)).cuda()
            key = (scene << 40 | first << 20 | second).sort().values
            first, second = key >> 20 & 0xfffff, key & 0xfffff
        else:
            key = (first << 32 | second).sort().values
            first, second = key >> 32, key & 0xffffffff
        pairs = torch.full((self.room, 2), -1, dtype=torch.int32, device="cuda")
        pairs[: len(key), 0], pairs[: len(key), 1] = first, second
        return pairs


def run(state):
    e, kind = engine(), state["kind"]
    if kind == "update":  # the boxes move there and, the next time, back
        scene = state["scene"]
        scene.move(state["idx"], state["next"])
        state["next"], state["after"] = state["after"], state["next"]
        removed, added = scene.delta(state["removed"], state["added"])
        return Found(state["room"], removed=removed, added=added, full=scene)
    stream, out = torch.cuda.current_stream(), state["out"]
    if kind == "batch":
        n = e.batch_intersect(state["boxes"], state["offsets"], state["range"], stream=stream)
        e.pairs_into(out[:n], stream=stream)
        return Found(len(out), pairs=out[:n], offsets=e.scene_offsets())
    e.set_pair_output(out)
    if kind == "redblue":
        n = e.bipartite_intersect(state["boxes"], state["blue"], state["range"], stream=stream)
    else:
        n = e.self_intersect(state["boxes"], state["range"], stream=stream)
    return Found(len(out), pairs=out[:n])


def work(case):
    """Each box read once, each pair (8 bytes) written once; an update reads the moved rows and
    writes the two lists of changed pairs and the full list after the move. Comparisons are not counted."""
    if case["kind"] == "update":
        changed = 2 * 1.96 * case["moved"]
        return {"bytes": case["moved"] * 32 + 8 * changed + 16 * _pairs_of(case), "flops": 0}
    if case["kind"] == "batch":
        n = sum(_sizes(case))
    else:
        n = case["n"] + case.get("n_blue", 0)
    row = 20 if case["kind"] == "plain2d" else 28
    return {"bytes": n * row + 8 * _pairs_of(case), "flops": 0}
