"""Totals of searches with more than 2^32 centres of one count: every centre of the area is in range, so
the total is known without a check."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", [0, 5])
@pytest.mark.parametrize("radius", [110_000, 125_000])
def test_total_counts_every_centre(radius, mode):
    from slime_b200.lib import SlimeCoreB200
    core = SlimeCoreB200()
    core.lib.slime_b200_set_engine(mode, 0)
    try:
        total, sites = core.search(90210, radius, 0, 221, 0, 0, 0, 1000)
    finally:
        core.lib.slime_b200_set_engine(0, 0)
    assert total == (2 * radius + 1) ** 2  # 4.8e10 and more: the fullest of the 222 counts has 9.3 % of them
    assert len(sites) == 1000 and sites["size"].min() >= 40
