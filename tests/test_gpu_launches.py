"""A small general scan is one launch at every threshold, also where no site is expected at all (shares down
to 1e-221: rows per launch worked out from them must not overflow)."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("radius", [0, 50, 300, 2000])
@pytest.mark.parametrize("low", [20, 36, 50, 62, 66, 80, 120, 221])
def test_one_launch(radius, low):
    from slime_b200.lib import SlimeCoreB200
    core = SlimeCoreB200()
    core.lib.slime_b200_set_engine(1, 0)
    try:
        core.lib.reset_cancel()
        core.search(90210, radius, low, 221, 0, 12_345, -67_890, 1000)
        assert core.last_search_stats()[1] == 1
    finally:
        core.lib.slime_b200_set_engine(0, 0)
