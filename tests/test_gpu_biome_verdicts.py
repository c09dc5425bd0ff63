"""The filter's verdict search (one bounded search per biome and quart column) against the biome ids of
every quart it stands for: all 16 columns of every slime chunk of each window, at the 17 Deep Dark
layers and the Mushroom Fields layer, for every vendored tree, both biome sizes and each flag."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DEEP_DARK, MUSHROOM = 183, 14
WINDOW = [(dx, dz) for dx in range(-8, 9) for dz in range(-8, 9) if dx * dx + dz * dz <= 68]


@pytest.fixture(scope="module")
def core():
    from slime_b200.lib import SlimeCoreB200
    return SlimeCoreB200()


@pytest.mark.parametrize("large", [0, 1])
@pytest.mark.parametrize("version", [1180, 1192, 1194, 1206, 1214, 1215, 2602])
def test_verdicts_equal_every_quart(core, version, large):
    from slime_b200.lib import BiomeFilter
    rng = np.random.Generator(np.random.PCG64(version + large))
    seed = int(rng.integers(-(2**63), 2**63, dtype=np.int64))
    n = 60
    cx = rng.integers(-1_800_000, 1_800_000, n).astype(np.int32)
    cz = rng.integers(-1_800_000, 1_800_000, n).astype(np.int32)
    x = np.concatenate([cx + dx for dx, _ in WINDOW])
    z = np.concatenate([cz + dz for _, dz in WINDOW])
    slime = core.is_slime_batch(seed, x, z).astype(bool)
    owner = np.tile(np.arange(n), len(WINDOW))[slime]
    qx = (4 * x[slime].astype(np.int64)[:, None] + np.arange(16) // 4).reshape(-1)
    qz = (4 * z[slime].astype(np.int64)[:, None] + np.arange(16) % 4).reshape(-1)
    owner = np.repeat(owner, 16)
    want = np.zeros(n, dtype=np.int32)
    with BiomeFilter(version, seed, len(qx), large=large, core=core) as f:
        for y in list(range(-16, 1)) + [16]:
            found = f.query(qx, np.full(len(qx), y), qz)
            if y == 16:
                want[owner[found == MUSHROOM]] |= 2
            else:
                want[owner[found == DEEP_DARK]] |= 1
        for flags in (1, 2, 3):
            assert np.array_equal(f.filter(cx, cz, flags), want & flags)
    if version >= 1192:  # 1.18 has no Deep Dark
        assert (want & 1).any()
