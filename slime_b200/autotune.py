"""Measure the engine crossovers of the slime-chunk search on the local GPU and write the rule.

    python -m slime_b200.autotune [--out slime_b200/tuning_b200.json] [--quick]

For each (radius, threshold) point of a grid the search is timed with every engine that applies
(the general scan, independent bands, and as columns in words and as bit planes grouped bands where the area
spans a period and the shared LCG where it spans two), forced through slime_b200_set_engine; every engine
must return the same total and the same ranked sites. From the timings it derives the twelve
numbers of slime_b200_set_engine_rule:

  band_min_threshold, band_min_periods   shared LCG from this threshold on areas this many
  band_fast_threshold, band_fast_periods 2^17-chunk periods wide (two branches of the rule)
  indep_min_threshold, indep_min_centres independent bands instead of the general scan
  exact_below_threshold, exact_min_centres  bit planes below this threshold on areas this large, where
                                         neither of the other band branches applies
  grouped_min_threshold, grouped_min_width, grouped_max_width
                                         grouped bands from this threshold on areas this wide
  exact_wide_below_threshold             bit planes below this threshold on areas 2.25+ periods wide

and writes them with the raw timings to a JSON file. SlimeCoreB200 applies that file when it
loads the library. The general scan's rate does not depend on the area once it fills the GPU, so
it is timed on the smaller areas only and extrapolated to the larger ones.
"""
from __future__ import annotations

import argparse
import ctypes
import json
import math
import time
from pathlib import Path

import numpy as np

PERIOD = 1 << 17
DEFAULT_OUT = Path(__file__).with_name("tuning_b200.json")
SEED = 0x5EED_B200  # any world seed: rates do not depend on it


def _time(core, mode, radius, thr, reps=2):
    core.lib.slime_b200_set_engine(mode, 0)
    best, out = None, None
    for _ in range(reps):
        core.lib.reset_cancel()
        t = time.perf_counter()
        out = core.search(SEED, radius, thr, 221, 0, 0, 0, 200)
        dt = time.perf_counter() - t
        best = dt if best is None else min(best, dt)
    return best, out


GROUPED_MAX_PERIODS = 16  # grouped bands hold at most 16 period copies
GROUPED_EXACT_MIN_WIDTH = 9 << 15  # the library's width from which bit planes run as grouped bands
GROUPED_SINGLE_MIN_WIDTH = 4 << 17  # and below SINGLE_BELOW, where windows are counted one by one
SINGLE_BELOW = 40
# The bit planes' branch has the thresholds below; only a batch's small searches would follow the
# independent bands' number there, and one alone is faster by the general scan (radius 2,000, threshold 40
# 0.14 ms, as independent bands 0.30).
INDEP_FROM = 42
BAND_MAX_SITES = 4e9  # expected sites that the band engines count
# On both sides of 8 and 16 periods, where a group more or less of copies fits a word.
RADII = [10_000, 30_000, 100_000, 150_000, 200_000, 300_000, 450_000, 520_000, 530_000, 600_000, 1_000_000,
         1_050_000, 1_250_000, 1_875_000]
THRESHOLDS = [40, 42, 44, 46, 48, 50, 52, 53, 54, 55, 56, 58, 60]


def tail_share(threshold):
    """Expected share of centres whose count reaches the threshold (221 cells, one in ten)."""
    return sum(math.comb(221, k) * 0.1**k * 0.9 ** (221 - k) for k in range(threshold, 222))


TAIL = [tail_share(t) for t in range(223)]


def engine(rule, width, threshold):
    """The engine that the library's rule picks for a full square (Context::engine_for), by its name in the
    timings; `rule` has the twelve numbers of slime_b200_set_engine_rule."""
    bt, bp, ft, fp, it, ic, et, ec, gt, gw, gx, ew = rule
    if width * width * TAIL[threshold] > BAND_MAX_SITES or threshold < 28:
        return "general"
    fits = width <= GROUPED_MAX_PERIODS * PERIOD
    wide = width >= GROUPED_EXACT_MIN_WIDTH
    shared = (threshold >= bt and width >= bp * PERIOD) or (threshold >= ft and width >= fp * PERIOD)
    grouped = threshold >= gt and width >= gw and fits and (width <= gx or not shared)
    if not shared and not grouped and threshold < (ew if wide else et) and width * width >= ec:
        if not wide or (threshold < SINGLE_BELOW and width < GROUPED_SINGLE_MIN_WIDTH):
            return "indep_exact" if threshold < SINGLE_BELOW else "indep"
        return "grouped_exact" if fits else "band_exact"
    if grouped:
        return "grouped"
    if shared:
        return "band"
    return "indep" if width * width >= ic and threshold >= it else "general"


def measure(core, quick=False):
    radii = [r for r in RADII if not quick or r <= 600_000]
    rows = []
    general_rate = {}
    for r in radii:
        w = 2 * r + 1
        for thr in THRESHOLDS[:: 2 if quick else 1]:
            point = {"radius": r, "threshold": thr, "centres": w * w}
            ref = None
            fits = w <= GROUPED_MAX_PERIODS * PERIOD
            engines = [("indep_exact", 5)]
            engines += [("band_exact", 4)] if w >= 2 * PERIOD else []
            engines += [("grouped_exact", 7)] if PERIOD < w and fits else []
            if thr >= 42 or r <= 100_000:  # bounded engines below 42 on large areas are never chosen
                engines += [("band", 2)] if w >= 2 * PERIOD else []
                engines += [("grouped", 6)] if PERIOD < w and fits else []
            if r <= 100_000:
                engines.insert(0, ("general", 1))
            for name, mode in engines:
                dt, out = _time(core, mode, r, thr, reps=2)
                if ref is None:
                    ref = out
                elif out[0] != ref[0] or not np.array_equal(out[1], ref[1]):
                    raise RuntimeError(f"engines disagree at radius {r} threshold {thr}")
                point[name + "_s"] = dt
            point["indep_s"] = point["indep_exact_s"]  # the same kernels
            if "general_s" in point:
                general_rate[thr] = point["centres"] / point["general_s"]
            else:
                point["general_s"] = point["centres"] / general_rate.get(thr, min(general_rate.values()))
            rows.append(point)
    core.lib.slime_b200_set_engine(0, 0)
    return rows


def planes_time(p):
    """Time of the bit planes in the mode that the library picks for the point; None if not timed."""
    w = 2 * p["radius"] + 1
    if w >= (GROUPED_SINGLE_MIN_WIDTH if p["threshold"] < SINGLE_BELOW else GROUPED_EXACT_MIN_WIDTH):
        for k in ("grouped_exact_s", "band_exact_s"):
            if k in p:
                return p[k]
    return p.get("indep_exact_s")


def planes_win(p):
    """Against the other branches of the rule (independent bands are the same kernels in both of theirs)."""
    return planes_time(p) < min(p[k] for k in ("general_s", "band_s", "grouped_s") if k in p)


def rule_time(p, rule):
    """Time of a point under a rule: infinite where the rule picks an engine that was not timed there."""
    name = engine(rule, 2 * p["radius"] + 1, p["threshold"])
    if name.endswith("_exact"):
        return planes_time(p) or math.inf
    return p.get(name + "_s", math.inf)


def best_time(p):
    return min(v for k, v in p.items() if k.endswith("_s"))


def derive(rows):
    """The rule numbers from the timings. Independent bands take a threshold when they beat
    the general scan there and at every higher measured threshold of the area. The two
    shared-LCG branches are chosen among the measured (threshold, periods) crossovers as the pair
    whose rule costs least over the whole grid (sum of each point's time over its best time), and
    the grouped-band branch (threshold, width range) is chosen the same way among the measured
    thresholds and widths. The costs are those of the rule that the library runs (engine)."""
    def min_winning_thr(pts, a, b):
        pts = sorted(pts, key=lambda p: p["threshold"])
        best = 222
        for p in reversed(pts):
            if a in p and b in p and p[a] < p[b]:
                best = p["threshold"]
            else:
                break
        return best

    by_r = {}
    for p in rows:
        if p["threshold"] >= INDEP_FROM:
            by_r.setdefault(p["radius"], []).append(p)
    indep_thr = {r: min_winning_thr(pts, "indep_s", "general_s") for r, pts in by_r.items()}
    indep_min_threshold = max(indep_thr.values())
    wins = [r for r, t in indep_thr.items() if t <= indep_min_threshold]
    indep = [indep_min_threshold, (2 * min(wins) + 1) ** 2 if wins else 1 << 62]
    exact, wide = derive_exact(rows), derive_exact_wide(rows)
    cands = sorted({(p["threshold"], max(2, (2 * p["radius"] + 1) // PERIOD)) for p in rows if "band_s" in p} | {(222, 64)})
    widths = sorted({2 * p["radius"] + 1 for p in rows if "grouped_s" in p})
    g_cands = [(t, lo, hi) for t in sorted({p["threshold"] for p in rows} | {222})
               for lo in widths for hi in widths if lo <= hi] or [(222, 1 << 40, 0)]
    best = [best_time(p) for p in rows]

    def numbers(a, b, g):
        return [*a, *b, *indep, *exact, *g, wide]

    def cost(a, b, g):
        rule = numbers(a, b, g)
        return sum(rule_time(p, rule) / t for p, t in zip(rows, best))

    # Coordinate descent: the shared-LCG pair without grouped bands, the grouped triple given the
    # pair, then the pair again given the triple.
    g = (222, 1 << 40, 0)
    pairs = [(x, y) for x in cands for y in cands if x <= y]
    a, b = min(pairs, key=lambda ab: cost(*ab, g))
    g = min(g_cands, key=lambda gg: cost(a, b, gg))
    a, b = min(pairs, key=lambda ab: cost(*ab, g))
    g = min(g_cands, key=lambda gg: cost(a, b, gg))
    return numbers(a, b, g)


def derive_exact(rows):
    """exact_below_threshold: one above the highest threshold at which the bit planes still beat every
    other branch on all areas of at least exact_min_centres centres, the smallest measured area where
    they win at the lowest threshold. (Wider areas have exact_wide_below_threshold.)"""
    pts = [p for p in rows if "indep_exact_s" in p and 2 * p["radius"] + 1 < GROUPED_EXACT_MIN_WIDTH]
    if not pts:
        return [0, 1 << 62]
    lowest = min(p["threshold"] for p in pts)
    winners = sorted(p["centres"] for p in pts if p["threshold"] == lowest and planes_win(p))
    if not winners:
        return [0, 1 << 62]
    min_centres = winners[0]
    below = 0
    for thr in sorted({p["threshold"] for p in pts}):
        big = [p for p in pts if p["threshold"] == thr and p["centres"] >= min_centres]
        if big and all(planes_win(p) for p in big):
            below = thr + 1
        else:
            break
    return [below, min_centres]


def derive_exact_wide(rows):
    """exact_wide_below_threshold: one above the highest threshold up to which the bit planes beat every
    other branch on some measured area at least GROUPED_EXACT_MIN_WIDTH wide: the library asks the other
    branches first, so that they keep the areas where they win."""
    pts = [p for p in rows if "indep_exact_s" in p and 2 * p["radius"] + 1 >= GROUPED_EXACT_MIN_WIDTH]
    below = 0
    for thr in sorted({p["threshold"] for p in pts}):
        at = [p for p in pts if p["threshold"] == thr]
        if any(planes_win(p) for p in at):
            below = thr + 1
        else:
            break
    return below


def main():
    ap = argparse.ArgumentParser()
    ap.add_argument("--out", default=str(DEFAULT_OUT))
    ap.add_argument("--quick", action="store_true", help="coarser grid (threshold step 4, no 1M radius)")
    ap.add_argument("--rederive", action="store_true", help="recompute the rule from the file's timings")
    args = ap.parse_args()
    from slime_b200 import build
    from slime_b200.lib import SlimeCoreB200
    build.build()
    core = SlimeCoreB200(apply_tuning=False)
    name = ctypes.create_string_buffer(256)
    core.lib.get_cuda_device_name(name, 256)
    device = name.value.decode(errors="replace")
    if args.rederive:
        old = json.loads(Path(args.out).read_text())
        rows, device = old["points"], old.get("device", device)
    else:
        rows = measure(core, quick=args.quick)
    rule = derive(rows)
    doc = {"device": device,
           "rule": dict(zip(["band_min_threshold", "band_min_periods", "band_fast_threshold",
                             "band_fast_periods", "indep_min_threshold", "indep_min_centres",
                             "exact_below_threshold", "exact_min_centres", "grouped_min_threshold",
                             "grouped_min_width", "grouped_max_width", "exact_wide_below_threshold"], rule)),
           "seed": SEED, "max_results": 200, "points": rows}
    Path(args.out).write_text(json.dumps(doc, indent=1) + "\n")
    print(json.dumps(doc["rule"]))


if __name__ == "__main__":
    main()
