"""The engine rule over widths and thresholds (no device needed): what the library picks where the branches
of the rule meet."""
import pytest

PERIOD = 1 << 17
GENERAL, SHARED, GROUPED, INDEPENDENT = 100, 200, 220, 300


@pytest.fixture(scope="module")
def core():
    from slime_b200 import build
    from slime_b200.lib import SlimeCoreB200
    build.build()
    core = SlimeCoreB200()
    core.lib.slime_b200_set_engine(0, 0)
    return core


def test_wide_areas_always_share_the_generator(core):
    """Areas several periods wide cost independent bands about twice the time of the modes that share work
    between periods: at no width and threshold may the branches leave a gap that sends them there."""
    radii = {int(147_456 * 1.02**i) for i in range(129)}
    for n in range(3, 29):  # on both sides of every period
        radii |= {(n * PERIOD - 1) // 2 + d for d in (-1, 0, 1)}
    radii |= {100_000 * k + d for k in range(2, 19) for d in (-1, 0, 1)} | {1_875_000}
    for r in sorted(r for r in radii if 147_456 <= r <= 1_875_000):
        for threshold in range(42, 90):
            assert core.lib.slime_b200_engine_for(r, threshold, 0) not in (GENERAL, INDEPENDENT), (r, threshold)


def test_grouped_bands_go_on_to_the_shared_lcg(core):
    for threshold in (56, 60, 75):
        for r in (500_000, 500_001, 510_000, 524_287):
            assert core.lib.slime_b200_engine_for(r, threshold, 0) == GROUPED
        assert core.lib.slime_b200_engine_for(524_288, threshold, 0) == SHARED


def test_a_disabled_branch_stays_off(core):
    before = core.engine_rule()
    try:
        core.set_engine_rule(dict(before, grouped_min_threshold=222))
        assert core.lib.slime_b200_engine_for(510_000, 60, 0) == INDEPENDENT
    finally:
        core.set_engine_rule(before)


def test_arguments_out_of_range(core):
    for args in ((-1, 40, 0), (10, 222, 0), (10, -1, 0), (10, 40, 11), (10, 40, -1), (2**31, 40, 0)):
        assert core.lib.slime_b200_engine_for(*args) == -1


def test_thin_annuli_of_low_thresholds_take_the_general_scan(core):
    pick = core.lib.slime_b200_engine_for
    for r, threshold in ((10_000, 28), (80_000, 29), (20_011, 30), (300_000, 35), (10_000, 36), (20_011, 39), (100_000, 38),
                         (147_456, 36), (200_000, 39), (400_000, 37), (690_000, 39), (150_000, 40), (900_000, 40)):
        line = 0.529 if threshold < 30 else 0.714 if threshold < 36 else 0.798 if threshold < 40 else 0.903
        inside, outside = line - 0.02, line + 0.02
        assert pick(r, threshold, int(outside * r)) == GENERAL
        assert pick(r, threshold, int(inside * r)) == pick(r, threshold, 0) != GENERAL
    for r in (147_456, 400_000, 900_000):
        for threshold in (41, 42, 50, 60):
            assert pick(r, threshold, r) == pick(r, threshold, 0) != GENERAL


def test_single_windows_of_narrow_areas_take_independent_bands(core):
    pick = core.lib.slime_b200_engine_for
    for r in (147_456, 200_000, 262_143):
        assert pick(r, 39, 0) == 310 and pick(r, 40, 0) == 230
    assert pick(262_144, 39, 0) == 230


def test_only_more_sites_than_the_bins_hold_leave_the_band_engines(core):
    """The band engines count a search into 32-bit bins, the general scan each of its launches."""
    pick = core.lib.slime_b200_engine_for
    assert pick(1_875_000, 40, 0) == pick(1_250_000, 40, 0) == 210  # 2.4e9 and 1.1e9 expected sites
    assert pick(1_875_000, 39, 0) == GENERAL                       # 4.9e9
    for mode in (2, 3, 4, 5, 6, 7):
        core.lib.slime_b200_set_engine(mode, 0)
        try:
            assert pick(1_875_000, 39, 0) == pick(125_000, 0, 0) == GENERAL
            assert pick(20_000, 40, 0) != GENERAL
        finally:
            core.lib.slime_b200_set_engine(0, 0)
