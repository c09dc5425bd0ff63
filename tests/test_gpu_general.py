"""The general scan against the oracle where its patches (240 x up to 128 centres) can go wrong: areas
one centre short of and past a patch's width, one or several rows a thread, a last patch of one row or
column, thresholds from 0, upper bounds, annuli, area corners at the int32 edge of block coordinates,
and Java's redraws (a seed that puts a redrawn slime chunk into the area). Results must be equal."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def core():
    from slime_b200.lib import SlimeCoreB200
    core = SlimeCoreB200()
    core.lib.slime_b200_set_engine(1, 0)
    yield core
    core.lib.slime_b200_set_engine(0, 0)


def check(core, oracle, seed, radius, low, high, inner, cx, cz, top):
    total, got = core.search(seed, radius, low, high, inner, cx, cz, top)
    want_total, want = oracle.search(seed, radius, low, high, inner, cx, cz, top)
    assert total == want_total
    assert np.array_equal(got, want)


# Widths 1, 7, 239, 241, 479, 481, 1,025: one to many patches, 1 to 4 rows a thread.
@pytest.mark.parametrize("radius", [0, 3, 119, 120, 239, 240, 512])
def test_patch_edges(core, oracle, radius):
    rng = np.random.Generator(np.random.PCG64(700 + radius))
    for low, high, inner in ((0, 221, 0), (30, 221, 0), (25, 30, radius // 2), (36, 221, radius)):
        seed = int(rng.integers(-(2**63), 2**63, dtype=np.int64))
        cx, cz = (int(v) for v in rng.integers(-1_800_000, 1_800_001, 2))
        check(core, oracle, seed, radius, low, high, inner, cx, cz, 2000)


def test_many_waves(core, oracle):
    check(core, oracle, 31337, 2500, 38, 221, 0, -250_001, 777_777, 5000)


@pytest.mark.parametrize("centre", [(2**31 - 200, -(2**31) + 200), (-(2**31) + 140, 2**31 - 140), (2**27, -(2**27))])
def test_coordinate_edges(core, oracle, centre):
    check(core, oracle, 99, 100, 30, 221, 0, *centre, 500)


def test_redrawn_chunk_in_the_area(core, oracle):
    """World seeds whose chunk (x, z) starts from a state that Java rejects and redraws into a slime
    chunk: state1 = 2^48 - k for small k."""
    mask, mul = (1 << 48) - 1, 0x5DEECE66D
    inverse = pow(mul, -1, 1 << 48)
    i32 = lambda v: (v & 0xFFFFFFFF) - ((v & 0x80000000) << 1)  # noqa: E731
    planted = 0
    for k in range(1, 400):
        state = (1 << 48) - k
        draw, bits = state, (1 << 31)
        while bits >= 2**31 - 8:
            draw = (draw * mul + 0xB) & mask
            bits = draw >> 17
        if bits % 10:
            continue
        x, z = 17 * k, -23 * k
        mix = ((state - 0xB) * inverse & mask) ^ mul ^ 0x3AD8025F
        mix -= i32(x * x * 0x4C1906) + i32(x * 0x5AC0DB) + i32(z * z) * 0x4307A7 + i32(z * 0x5F24F)
        seed = mix & mask
        assert oracle.is_slime(seed, x, z)
        check(core, oracle, seed, 30, 20, 221, 0, x + 5, z - 3, 4000)
        planted += 1
        if planted == 5:
            break
    assert planted == 5
