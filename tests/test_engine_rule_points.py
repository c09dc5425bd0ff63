"""The committed engine rule against the timings it is committed with, and the tuner's form of the rule
against the library's."""
import itertools
import json

import pytest

from slime_b200.autotune import PERIOD, best_time, derive, engine, rule_time
from slime_b200.lib import RULE_KEYS, TUNING

NAMES = {100: "general", 200: "band", 210: "band_exact", 220: "grouped", 230: "grouped_exact", 300: "indep",
         310: "indep_exact"}


@pytest.fixture(scope="module")
def doc():
    return json.loads(TUNING.read_text())


@pytest.fixture(scope="module")
def core():
    from slime_b200 import build
    from slime_b200.lib import SlimeCoreB200
    build.build()
    core = SlimeCoreB200(apply_tuning=False)
    core.lib.slime_b200_set_engine(0, 0)
    return core


def test_the_rule_follows_from_its_points(doc, core):
    assert derive(doc["points"]) == [doc["rule"][k] for k in RULE_KEYS]
    assert core.engine_rule() == doc["rule"]  # the library's defaults


def test_the_rule_is_near_the_best_time_at_every_point(doc):
    rule = [doc["rule"][k] for k in RULE_KEYS]
    for p in doc["points"]:
        assert rule_time(p, rule) <= 1.1 * best_time(p), (p["radius"], p["threshold"])


def test_between_the_points_the_rule_picks_what_wins_beside_them(doc):
    """At any width and timed threshold: an engine within 12 % of the best at the nearest narrower or the
    nearest wider radius that was timed (the two sides of a line may differ)."""
    rule = [doc["rule"][k] for k in RULE_KEYS]
    radii = sorted({p["radius"] for p in doc["points"]})
    points = {(p["radius"], p["threshold"]): p for p in doc["points"]}
    for threshold in sorted({t for _, t in points}):
        for lo, hi in zip(radii, radii[1:]):
            for k in range(1, 40):
                r = int(lo * (hi / lo) ** (k / 40))
                name = engine(rule, 2 * r + 1, threshold)
                sides = [points[s, threshold] for s in (lo, hi)]
                assert any(p.get(name + "_s", 1e9) <= 1.12 * best_time(p) for p in sides), (r, threshold, name)


def test_the_tuner_scores_the_rule_that_the_library_runs(core):
    widths = {2 * r + 1 for r in (100, 9_999, 10_000, 40_000, 100_000, 147_455, 147_456, 262_143, 262_144, 300_000,
                                  500_000, 524_287, 524_288, 1_000_000, 1_048_575, 1_048_576, 1_875_000, 40_000_000)}
    rules = [[53, 16, 55, 8, 42, 400040001, 55, 400040001, 55, 200001, 1000001, 55],
             [44, 15, 44, 15, 42, 400040001, 45, 400040001, 46, 200001, 2000001, 45],
             [222, 64, 222, 64, 40, 0, 0, 0, 222, 0, 0, 0],
             [60, 2, 50, 4, 48, 10**10, 60, 10**11, 52, 300_001, 600_001, 50]]
    before = core.engine_rule()
    try:
        for rule in rules:
            core.set_engine_rule(dict(zip(RULE_KEYS, rule)))
            for width, threshold in itertools.product(widths, (0, 27, 28, 35, 39, 40, 41, 43, 44, 47, 52, 55, 61, 221)):
                got = core.lib.slime_b200_engine_for((width - 1) // 2, threshold, 0)
                assert NAMES[got] == engine(rule, width, threshold), (rule, width, threshold)
    finally:
        core.set_engine_rule(before)
    assert PERIOD == 1 << 17


def test_the_binding_reads_the_rule_of_the_file(doc, core, tmp_path):
    from slime_b200.lib import SlimeCoreB200, tuned_rule
    assert tuned_rule() == doc["rule"]
    other = tmp_path / "rule.json"
    other.write_text(json.dumps({"rule": dict(doc["rule"], band_min_threshold=60), "points": []}, indent=2))
    assert tuned_rule(other) == dict(doc["rule"], band_min_threshold=60)
    before = core.engine_rule()
    try:
        core.set_engine_rule(dict(before, band_min_threshold=60))
        assert SlimeCoreB200().engine_rule() == doc["rule"]
    finally:
        core.set_engine_rule(before)
