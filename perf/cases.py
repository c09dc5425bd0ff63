"""Timed cases of the slime-chunk cluster search, through the public Python binding.

Each case is one call (or one small set of calls) that a frontend or a service makes:

  search   SlimeCoreB200.search: one seed, one square or annulus of centres, ranked sites
  batch    SlimeCoreB200.search_batch: many seeds in one call
  serve    SlimeServer: a burst of requests submitted, waited for and taken
  filter   BiomeFilter.filter: Deep Dark / Mushroom Fields verdicts of candidate sites
  score    SlimeCoreB200.score_precise: precise AFK scores of ranked sites

Sizes follow slime_b200/workloads.py (the 4,001^2 search, the mixed batch, the served stream, scores
and biome verdicts of every site) and the radii and thresholds of slime_b200/tuning_b200.json. Inputs
and results live in host memory, as the C ABI takes them. All outputs are whole numbers.
"""
import math

import numpy as np

from slime_b200.lib import RESULT_DTYPE, BiomeFilter, SlimeCoreB200, SlimeServer
from slime_b200.workloads import Search

WORLD = 1_875_000  # world border in chunks


def _search(name, radius, min_size, max_results=1000, **more):
    return dict({"kind": "search", "radius": radius, "min_size": min_size, "max_results": max_results,
                 "rd_min": 0, "max_size": 221, "precise": 0}, name=name, **more)


def listed():
    return [
        # A look around one base: the smallest request of the served stream; launch latency.
        _search("search r100 t36", 100, 36),
        # The reference's own example search: 4,001^2 centres, every site wanted.
        _search("search r2000 t40", 2000, 40, 100_000),
        # Sites away from spawn: an annulus with precise AFK scores of the best 100.
        _search("search r9001 t44 annulus afk", 9001, 44, 1000, rd_min=3000, precise=1),
        # An ordinary search: tens of thousands of chunks, a rare site size.
        _search("search r20011 t50", 20_011, 50),
        # Every good site of a large region: a low threshold.
        _search("search r100000 t42", 100_000, 42),
        # The best sites of a large region: a high threshold on an area a few periods wide.
        _search("search r200000 t53", 200_000, 53),
        # A low threshold on an area several periods wide.
        _search("search r300000 t44", 300_000, 44),
        # The largest: two thirds of the world's width at the headline threshold.
        _search("search r1250000 t60", 1_250_000, 60),
        # Scanning seeds: one call with the mixed radii and thresholds of the 64-seed batch, up to 5e4.
        {"name": "batch 16 r1000-50000", "kind": "batch", "count": 16, "radius_lo": 1000, "radius_hi": 50_000},
        # A burst at the search server: small and medium requests, a quarter of them biome-filtered.
        {"name": "serve 24 r100-50000", "kind": "serve", "count": 24, "radius_lo": 100, "radius_hi": 50_000},
        # Biome exclusion of the ranked sites of one search (both biomes, Minecraft 26.2).
        {"name": "filter 4096 sites", "kind": "filter", "sites": 4096, "flags": 3, "version": 2602},
        # Precise AFK scores of every site of a search.
        {"name": "score 20000 sites", "kind": "score", "sites": 20_000, "y_scan": 0},
    ]


def _log_uniform(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["search", "search", "search", "search", "batch", "serve", "filter", "score"])
    if kind == "search":
        # A threshold that some sites of the area reach (the share of centres falls 2.4-fold per
        # unit, from 1.7e-4 at 40). Low thresholds cost more per centre: their areas end earlier, so
        # that no draw costs more than the largest listed case.
        r = _log_uniform(rng, 100, 1_250_000)
        high = 40 + int((2 * math.log10(2 * r + 1) - 5.1) / 0.385)
        t = rng.randint(36 if r < 4000 else 40 if r < 300_000 else 46 if r < 500_000 else 58, high)
        return {"kind": kind, "radius": r, "min_size": t, "max_results": rng.choice([100, 1000, 10_000]),
                "rd_min": rng.choice([0, 0, 0, r // 3]), "max_size": rng.choice([221, 221, 221, t + 4]),
                "precise": rng.choice([0, 0, 1])}
    if kind in ("batch", "serve"):
        return {"kind": kind, "count": rng.randint(8, 32), "radius_lo": 1000 if kind == "batch" else 100,
                "radius_hi": _log_uniform(rng, 10_000, 50_000)}
    if kind == "filter":
        return {"kind": kind, "sites": _log_uniform(rng, 100, 8000), "flags": rng.choice([1, 2, 3, 3]),
                "version": rng.choice([1194, 1206, 2105, 2602])}
    return {"kind": kind, "sites": _log_uniform(rng, 100, 40_000) if rng.random() < 0.7 else rng.randint(100, 1000),
            "y_scan": rng.choice([0, 0, 1])}


def _world_seed(rng):
    return int(rng.integers(-(2**63), 2**63, dtype=np.int64))


def _requests(case, rng):
    """Seeded requests with the distributions of the batch and of the served stream."""
    out = []
    for _ in range(case["count"]):
        r = int(round(math.exp(rng.uniform(math.log(case["radius_lo"]), math.log(case["radius_hi"])))))
        serve = case["kind"] == "serve"
        t = int(rng.integers(40, 66)) if serve else int(rng.integers(45, 61))
        out.append(Search(seed=_world_seed(rng), center_x=int(rng.integers(-1_000_000, 1_000_001)),
                          center_z=int(rng.integers(-1_000_000, 1_000_001)), radius=r, min_size=t,
                          biome_flags=3 if serve and rng.uniform() < 0.25 else 0))
    return out


def _sites(core, seed, n):
    """The best n sites of a search wide enough to have them (2e-5 of the centres reach 44)."""
    radius = max(2000, int(math.sqrt(n / 2e-5)))
    core.lib.reset_cancel()
    total, sites = core.search(seed, radius, 44, max_results=n)
    return sites


class _Serving:
    """A server that stops with the last reference to it."""

    def __init__(self, core):
        self.server = SlimeServer(core=core)

    def __del__(self):
        self.server.close()


class _Filter:
    def __init__(self, core, version, seed, capacity):
        self.filter = BiomeFilter(version, seed, capacity, core=core)

    def __del__(self):
        self.filter.close()


def _generator(case, seed):
    return np.random.Generator(np.random.PCG64([seed, 0x511E, sum(map(ord, case["kind"]))]))


def _centre(case, rng):
    room = min(WORLD, 1_000_000) if case["radius"] < 500_000 else max(0, WORLD - case["radius"])
    return int(rng.integers(-room, room + 1)), int(rng.integers(-room, room + 1))


def prepare(case, seed):
    rng = _generator(case, seed)
    core = SlimeCoreB200()
    state = {"case": case, "core": core, "seed": _world_seed(rng)}
    if case["kind"] == "search":
        state["centre"] = _centre(case, rng)
    elif case["kind"] in ("batch", "serve"):
        state["requests"] = _requests(case, rng)
        if case["kind"] == "serve":
            state["serving"] = _Serving(core)
    else:
        sites = _sites(core, state["seed"], case["sites"])
        if case["kind"] == "score":
            state["sites"] = sites
        else:
            state["cx"] = (sites["center_x"] - 8) // 16
            state["cz"] = (sites["center_z"] - 8) // 16
            state["filter"] = _Filter(core, case["version"], state["seed"], max(len(sites), 1))
    return state


def _numbers(records):
    """Result records as rows of six whole numbers."""
    return records.view(np.int32).reshape(*records.shape, len(RESULT_DTYPE.names))


def _gather(done, requests):
    """(total, sites) of many requests as their totals and one row of max_results records each."""
    totals = np.array([total for total, _ in done], dtype=np.int64)
    rows = np.zeros((len(requests), max(q.max_results for q in requests)), dtype=RESULT_DTYPE)
    for row, (_, sites) in zip(rows, done):
        row[: len(sites)] = sites
    return [totals, _numbers(rows)]


def run(state):
    case, core = state["case"], state["core"]
    kind = case["kind"]
    if kind == "search":
        if case["precise"]:
            core.set_y_scan_config(0)
        sites = np.zeros(case["max_results"], dtype=RESULT_DTYPE)
        total, _ = core.search(state["seed"], case["radius"], case["min_size"], case["max_size"], case["rd_min"],
                               *state["centre"], case["max_results"], case["precise"], out=sites)
        return [total, _numbers(sites)]
    if kind == "batch":
        return _gather(core.search_batch(state["requests"]), state["requests"])
    if kind == "serve":
        server = state["serving"].server
        tickets = [server.submit(q) for q in state["requests"]]
        done = []
        for ticket, q in zip(tickets, state["requests"]):
            server.wait(ticket)
            done.append(server.take(ticket, q.max_results)[:2])
        return _gather(done, state["requests"])
    if kind == "filter":
        return state["filter"].filter.filter(state["cx"], state["cz"], case["flags"])
    core.set_y_scan_config(case["y_scan"])
    return _numbers(core.score_precise(state["seed"], state["sites"]))


def work(case):
    """Whole-number operations a pass cannot do without, and the records in and out."""
    kind = case["kind"]
    if kind == "search":
        inner = math.pi * case["rd_min"] ** 2
        centres = (2 * case["radius"] + 1) ** 2 - inner
        return {"bytes": 24 * case["max_results"] + 48, "flops": 4 * centres}  # one first-draw test per centre
    if kind in ("batch", "serve"):
        # Mean area of a log-uniform radius.
        lo, hi = case["radius_lo"], case["radius_hi"]
        mean = 4 * (hi**2 - lo**2) / (2 * math.log(hi / lo))
        return {"bytes": 56 * case["count"] + 24 * 1000 * case["count"], "flops": 4 * mean * case["count"]}
    if kind == "filter":
        # About 20 slime chunks of their own per site, 16 quart columns each: 52 Perlin samples.
        return {"bytes": 12 * case["sites"], "flops": case["sites"] * 20 * 16 * 52 * 60}
    # 44 slime chunks in reach of each of 81 positions, at 1 or 33 heights.
    return {"bytes": 48 * case["sites"], "flops": case["sites"] * 81 * 44 * (33 if case["y_scan"] else 1)}


def _slime(seed, x, z):
    """Slime chunks of the grid z (rows) by x (columns): Java's Random in wrapping 64-bit arithmetic."""
    i32 = lambda v: (v & 0xFFFFFFFF).astype(np.int32).astype(np.int64)  # noqa: E731
    xt = i32(x * x * 0x4C1906) + i32(x * 0x5AC0DB)
    zt = i32(z * z) * 0x4307A7 + i32(z * 0x5F24F)
    mask = (1 << 48) - 1
    with np.errstate(over="ignore"):
        state = (((xt[None, :] + (zt + np.int64(seed))[:, None]) ^ 0x3AD8025F) ^ 0x5DEECE66D) & mask
        slime = np.zeros(state.shape, dtype=bool)
        todo = np.ones(state.shape, dtype=bool)
        while todo.any():
            state[todo] = (state[todo] * 0x5DEECE66D + 0xB) & mask
            bits = state[todo] >> 17
            value = bits % 10
            final = bits - value + 9 < 1 << 31
            at = np.flatnonzero(todo)
            slime.reshape(-1)[at[final]] = value[final] == 0
            todo.reshape(-1)[at[final]] = False
    return slime


def exact(case, seed):
    """The searches of up to 2e7 centres without scores, in plain numpy."""
    if case["kind"] != "search" or case["precise"] or (2 * case["radius"] + 1) ** 2 > 2e7:
        return None
    rng = _generator(case, seed)
    world = _world_seed(rng)
    cx, cz = _centre(case, rng)
    r, n = case["radius"], 2 * case["radius"] + 1
    off = np.arange(-r - 8, r + 9, dtype=np.int64)
    grid = _slime(world, cx + off, cz + off).astype(np.int16)
    count = np.zeros((n, n), dtype=np.int16)
    for dz in range(-8, 9):
        for dx in range(-8, 9):
            if dx * dx + dz * dz <= 68:
                count += grid[8 + dz:8 + dz + n, 8 + dx:8 + dx + n]
    keep = (count >= case["min_size"]) & (count <= case["max_size"])
    if case["rd_min"]:
        d = np.arange(-r, r + 1, dtype=np.int64) ** 2
        keep &= d[:, None] + d[None, :] >= case["rd_min"] ** 2
    z, x = np.nonzero(keep)
    size, bx, bz = count[z, x].astype(np.int64), 16 * (cx - r + x) + 8, 16 * (cz - r + z) + 8
    order = np.lexsort((bz, bx, -size))[: case["max_results"]]
    size, bx, bz = size[order], bx[order], bz[order]
    rows = np.zeros((case["max_results"], 6), dtype=np.int32)
    rows[: len(size)] = np.stack([size, bx, bz, np.zeros_like(size), bx, bz], axis=1)
    return [len(x), rows]
