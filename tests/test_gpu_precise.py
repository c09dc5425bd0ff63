"""The one-level precise scoring kernel against the oracle: one site to several rounds of a CTA, sites of
all 16 alignments mixed in one call (search results have one), both offset scans, packed and plain
scores, and sites at the int32 edge. Whole numbers: results must be equal."""
import numpy as np
import pytest

from oracle.oracle import YConfig

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def core():
    from slime_b200.lib import SlimeCoreB200
    core = SlimeCoreB200()
    core.set_y_scan_config(0, -64, -64, 64, 4)
    return core


def sites(rng, n, aligned):
    from slime_b200.lib import RESULT_DTYPE
    out = np.zeros(n, dtype=RESULT_DTYPE)
    for f in ("center_x", "center_z"):
        v = rng.integers(-30_000_000, 30_000_001, n)
        out[f] = v // 16 * 16 + 8 if aligned else v
    out["size"] = 40
    out["afk_x"], out["afk_z"] = out["center_x"], out["center_z"]
    return out


@pytest.mark.parametrize("scan_xz", [0, 1])
@pytest.mark.parametrize("n,aligned", [(1, True), (7, False), (593, True), (600, False), (5000, True)])
def test_scores_match_the_oracle(core, oracle, n, aligned, scan_xz):
    rng = np.random.Generator(np.random.PCG64(40 * n + scan_xz))
    seed = int(rng.integers(-(2**63), 2**63, dtype=np.int64))
    s = sites(rng, n, aligned)
    assert np.array_equal(core.score_precise(seed, s, scan_xz), oracle.score_precise(seed, s, scan_xz))


def test_other_platform_levels_and_edges(core, oracle):
    rng = np.random.Generator(np.random.PCG64(5))
    s = sites(rng, 40, False)
    s["center_x"][:4] = [2**31 - 300, -(2**31) + 300, 0, -1]
    for platform in (-64, 70):
        core.set_y_scan_config(0, platform, -64, 64, 4)
        try:
            got = core.score_precise(77, s, 1)
        finally:
            core.set_y_scan_config(0, -64, -64, 64, 4)
        assert np.array_equal(got, oracle.score_precise(77, s, 1, YConfig(0, platform, -64, 64, 4)))
