"""Ranking when far more sites share the lowest count that ranks than can be returned: an upper bound stops
the emission gate there. The best of the threshold's sites must come in order, ties by block x, then z."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def core():
    from slime_b200.lib import SlimeCoreB200
    return SlimeCoreB200()


# (radius, low, high, mode): 64 and more ties for each ranked site, and few of them
@pytest.mark.parametrize("radius,low,high,mode", [(700, 30, 31, 5), (700, 30, 31, 7), (1200, 28, 28, 5), (300, 30, 33, 5)])
@pytest.mark.parametrize("top", [1, 2, 63, 64, 100, 1000, 5000])
def test_ties_at_the_gate(core, oracle, radius, low, high, mode, top):
    core.lib.slime_b200_set_engine(mode, 0)
    try:
        total, got = core.search(31337, radius, low, high, 0, 4_000, -9_000, top)
    finally:
        core.lib.slime_b200_set_engine(0, 0)
    want_total, want = oracle.search(31337, radius, low, high, 0, 4_000, -9_000, top)
    assert total == want_total
    assert np.array_equal(got, want)


def test_ties_where_block_coordinates_wrap(core, oracle):
    """Past 2^27 chunks the order is that of wrapped 32-bit block coordinates."""
    core.lib.slime_b200_set_engine(5, 0)
    try:
        total, got = core.search(99, 400, 30, 31, 0, 2**27, -(2**27), 50)
    finally:
        core.lib.slime_b200_set_engine(0, 0)
    want_total, want = oracle.search(99, 400, 30, 31, 0, 2**27, -(2**27), 50)
    assert total == want_total
    assert np.array_equal(got, want)


@pytest.mark.parametrize("radius,low,high,mode", [(6000, 26, 27, 5), (6000, 26, 27, 7), (6000, 27, 27, 4)])
def test_more_sites_at_the_gate_than_the_hit_buffer_holds(core, radius, low, high, mode):
    """Five million sites share the highest count in range; the general scan is the check."""
    results = []
    for m in (1, mode):
        core.lib.slime_b200_set_engine(m, 0)
        try:
            results.append(core.search(-5, radius, low, high, 0, 77_000, 1_000, 20_000))
        finally:
            core.lib.slime_b200_set_engine(0, 0)
    assert results[0][0] == results[1][0]
    assert np.array_equal(results[0][1], results[1][1])


@pytest.mark.parametrize("low,high,engine", [(30, 33, 100), (36, 37, 100), (39, 221, 310), (40, 44, 300), (45, 45, 300)])
def test_searches_that_send_many_sites_take_the_general_scan(core, low, high, engine):
    """Radius 12,000: an upper bound that leaves many sites at the best count (0.6 % and 0.06 % of the centres),
    and bounds that do not."""
    total, got = core.search(77, 12_000, low, high, 0, 1_000, -1_000, 500)
    assert core.lib.get_gpu_v1_algorithm() == engine
    core.lib.slime_b200_set_engine(5, 0)
    try:
        total5, got5 = core.search(77, 12_000, low, high, 0, 1_000, -1_000, 500)
    finally:
        core.lib.slime_b200_set_engine(0, 0)
    assert total == total5
    assert np.array_equal(got, got5)
