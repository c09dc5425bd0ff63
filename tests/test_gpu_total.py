"""Totals of searches with more than 2^32 centres of one count: every centre of the area is in range, so
the total is known without a check."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("radius", [110_000, 125_000])
def test_total_counts_every_centre(radius):
    from slime_b200.lib import SlimeCoreB200
    core = SlimeCoreB200()
    total, sites = core.search(90210, radius, 0, 221, 0, 0, 0, 1000)
    assert total == (2 * radius + 1) ** 2  # 4.8e10 and more: the fullest of the 222 counts has 9.3 % of them
    assert len(sites) == 1000 and sites["size"].min() >= 40
