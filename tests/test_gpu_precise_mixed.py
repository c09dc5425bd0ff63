"""One-level scores of sites of several alignments (centres that are not 8 mod 16): chunks of one class, of
several, and of one with a stranger in their last place, against the oracle; and their time beside that of as
many search results."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def core():
    from slime_b200.lib import SlimeCoreB200
    core = SlimeCoreB200()
    core.set_y_scan_config(0, -64, -64, 64, 4)
    return core


def sites(x, z):
    from slime_b200.lib import RESULT_DTYPE
    out = np.zeros(len(x), dtype=RESULT_DTYPE)
    out["center_x"], out["center_z"], out["size"] = x, z, 40
    return out


@pytest.mark.parametrize("scan_xz", [0, 1])
@pytest.mark.parametrize("n", [2, 8, 9, 600, 1184, 1185, 4737, 6000])
@pytest.mark.parametrize("kind", ["runs", "stranger", "mixed"])
def test_scores_of_mixed_alignments(core, oracle, n, kind, scan_xz):
    rng = np.random.Generator(np.random.PCG64(100 * n + scan_xz))
    x, z = (rng.integers(-1_000_000, 1_000_001, n) * 16 + 8 for _ in range(2))
    if kind == "runs":  # 100 sites of a class, then the next
        x, z = x + np.arange(n) // 100 % 4, z + np.arange(n) // 400 % 4
    elif kind == "stranger":
        x[7::8] += 1
        x[-1] += 2
    else:
        x, z = x + rng.integers(0, 16, n), z + rng.integers(0, 16, n)
    s = sites(x, z)
    assert np.array_equal(core.score_precise(-12, s, scan_xz), oracle.score_precise(-12, s, scan_xz))


def test_mixed_alignments_cost_little_more(core):
    """Lookups in global memory instead of a table for every class of a chunk (1.6 times the aligned sites')."""
    rng = np.random.Generator(np.random.PCG64(8))
    x, z = (rng.integers(-1_000_000, 1_000_001, 5000) * 16 + 8 for _ in range(2))
    best = {}
    for name, s in (("aligned", sites(x, z)), ("mixed", sites(x + rng.integers(0, 16, 5000), z))):
        runs = []
        for _ in range(40):
            t0 = time.perf_counter()
            core.score_precise(-12, s, 1)
            runs.append(time.perf_counter() - t0)
        best[name] = min(runs)
    assert best["mixed"] < 1.4 * best["aligned"], best
