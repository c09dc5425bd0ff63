"""The bit-plane band kernels (exact counts in every band mode, bounded independent bands) against the
oracle at the edges of their tiles: areas one centre short of and past one tile's 1,008 (shared LCG:
496) columns, heights that leave a batch or a strip unfinished, single rows a band, annuli, upper
bounds and the smallest areas. Whole numbers: results must be equal."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def core():
    from slime_b200.lib import SlimeCoreB200
    return SlimeCoreB200()


# radius: widths 1, 17, 81 (below 8 rows a band), 495 / 497, 1,007 / 1,009, 1,483
@pytest.mark.parametrize("radius", [0, 8, 40, 247, 248, 503, 504, 741])
@pytest.mark.parametrize("mode", [3, 4, 5, 7])
def test_plane_kernels_match_the_oracle(core, oracle, mode, radius):
    rng = np.random.Generator(np.random.PCG64(9000 + 10 * radius + mode))
    for low, high, inner in ((28, 221, 0), (33, 221, 0), (30, 36, radius // 2)):
        seed = int(rng.integers(-(2**63), 2**63, dtype=np.int64))
        cx, cz = (int(v) for v in rng.integers(-1_800_000, 1_800_001, 2))
        core.lib.slime_b200_set_engine(mode, 0)
        try:
            total, got = core.search(seed, radius, low, high, inner, cx, cz, 3000)
        finally:
            core.lib.slime_b200_set_engine(0, 0)
        want_total, want = oracle.search(seed, radius, low, high, inner, cx, cz, 3000)
        assert total == want_total
        assert np.array_equal(got, want)


@pytest.mark.parametrize("mode", [5, 7])
def test_exact_counts_of_every_centre(core, oracle, mode):
    """Threshold 0: every centre is in range, so every count of the area is checked."""
    core.lib.slime_b200_set_engine(mode, 0)
    try:
        total, got = core.search(-77, 60, 0, 221, 0, 1_000_003, -999_983, 121 * 121)
    finally:
        core.lib.slime_b200_set_engine(0, 0)
    want_total, want = oracle.search(-77, 60, 0, 221, 0, 1_000_003, -999_983, 121 * 121)
    assert total == want_total == 121 * 121
    assert np.array_equal(got, want)


# Modes 6 and 7 on areas of 1.2 to 4.6 periods: 8, 5, 4 and 3 groups of copies; 5 and 3 do not divide
# the period. Independent bands, which share nothing, are the check.
@pytest.mark.parametrize("radius", [80_000, 140_000, 200_000, 270_000])
def test_groups_of_copies_match_independent_bands(core, radius):
    results = []
    for mode in (7, 5):
        core.lib.slime_b200_set_engine(mode, 0)
        try:
            results.append(core.search(4242, radius, 50, 221, 0, -31_337, 65_537, 2000))
        finally:
            core.lib.slime_b200_set_engine(0, 0)
    assert results[0][0] == results[1][0]
    assert np.array_equal(results[0][1], results[1][1])
