"""Low thresholds on the bit planes: what is done for each centre that is kept (1 to 3 in 1,000 here) must
stay small beside generating and counting. Grouped bands share the generator's work and test fewer chunks
than independent bands on these areas; with the same kept centres they cannot be much slower."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("radius,low", [(180_000, 36), (180_000, 38), (270_000, 37)])
def test_kept_centres_of_grouped_bands_cost_little(radius, low):
    from slime_b200.lib import SlimeCoreB200
    core = SlimeCoreB200()
    times, results = {}, {}
    for mode in (5, 7):
        core.lib.slime_b200_set_engine(mode, 0)
        try:
            runs = []
            for _ in range(3):
                core.lib.reset_cancel()
                results[mode] = core.search(20240607, radius, low, 221, 0, 3000, -77, 1000)
                runs.append(core.last_search_stats()[0])
            times[mode] = min(runs)
        finally:
            core.lib.slime_b200_set_engine(0, 0)
    assert results[5][0] == results[7][0]
    assert np.array_equal(results[5][1], results[7][1])
    # 1.1 to 1.25 times the independent bands' time; 2 to 2.2 with the bands' rows divided out for each centre.
    assert times[7] < 1.4 * times[5]


# The rule's choice against the modes it passes over, where its branches meet. General scans of whole wide
# areas (mode 1) are left out: they are never near.
@pytest.mark.parametrize("radius,low,inner,modes", [
    (510_000, 60, 0, (2, 3, 6, 7)), (524_287, 56, 0, (2, 3, 6, 7)), (524_288, 58, 0, (2, 3, 6, 7)),
    (200_000, 38, 150_000, (1, 4, 5, 7)), (200_000, 38, 180_000, (1, 4, 5, 7)), (400_000, 39, 396_000, (1, 4, 5, 7)),
])
def test_the_rule_is_near_the_fastest_mode(radius, low, inner, modes):
    from slime_b200.lib import SlimeCoreB200
    core = SlimeCoreB200()
    times, results = {}, {}
    for mode in (0,) + modes:
        core.lib.slime_b200_set_engine(mode, 0)
        try:
            runs = []
            for _ in range(2):
                core.lib.reset_cancel()
                results[mode] = core.search(20240607, radius, low, 221, inner, 3000, -77, 1000)
                runs.append(core.last_search_stats()[0])
            times[mode] = min(runs)
        finally:
            core.lib.slime_b200_set_engine(0, 0)
        assert results[mode][0] == results[0][0] and np.array_equal(results[mode][1], results[0][1]), mode
    assert times[0] < 1.15 * min(times[mode] for mode in modes), times


def test_an_upper_bound_does_not_scan_twice():
    """Ten million sites share the highest count in range of counts 38 to 40, and all are sent: launches sized
    to the hit buffer instead of run again in halves (1.15 times the time without the bound, 2.9 before)."""
    from slime_b200.lib import SlimeCoreB200
    core = SlimeCoreB200()
    times = {}
    for high in (221, 40):
        runs = []
        for _ in range(2):
            core.lib.reset_cancel()
            core.search(20240607, 200_000, 38, high, 0, 3000, -77, 1000)
            runs.append(core.last_search_stats()[0])
        times[high] = min(runs)
    assert times[40] < 1.6 * times[221], times
