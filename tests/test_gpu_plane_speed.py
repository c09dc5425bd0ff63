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
