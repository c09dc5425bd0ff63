"""The bit-plane kernels that count 2 or 4 adjacent windows as one, against the oracle where they can go wrong:
sites in the first and last columns and rows of the area and of a tile (1,008 columns; shared LCG 496), at every
row of a batch, upper bounds and annuli; and at thresholds so low that the list of unions (1,024 a batch)
overflows and the warps count what is left themselves. Whole numbers: results must be equal."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def core():
    from slime_b200.lib import SlimeCoreB200
    core = SlimeCoreB200()
    yield core
    core.lib.slime_b200_set_engine(0, 0)
    core.lib.slime_b200_set_plane_union(0)


def run(core, mode, joined, *case):
    core.lib.slime_b200_set_engine(mode, 0)
    core.lib.slime_b200_set_plane_union(joined)
    try:
        return core.search(*case)
    finally:
        core.lib.slime_b200_set_engine(0, 0)
        core.lib.slime_b200_set_plane_union(0)


@pytest.fixture(scope="module")
def rich(oracle):
    """A site of 49 or more and its seed."""
    for seed in range(1, 40):
        total, sites = oracle.search(seed, 3000, 49, 221, 0, 0, 0, 10)
        if total:
            return seed, int(sites["center_x"][0] - 8) // 16, int(sites["center_z"][0] - 8) // 16
    raise AssertionError("no site of 49 found")


# Unforced, unions of four at 47 and above, of two at 40: the site in the area's column `u` and row `v`.
@pytest.mark.parametrize("mode", [3, 4, 5, 7])
@pytest.mark.parametrize("low", [40, 47])
@pytest.mark.parametrize("u,v", [(0, 0), (1, 5), (2, 6), (3, 11), (494, 1), (495, 2), (496, 3), (497, 4), (1006, 7),
                                 (1007, 8), (1008, 9), (1009, 10), (1240, 1240), (1237, 1239), (600, 38), (601, 39)])
def test_sites_at_tile_edges(core, oracle, rich, mode, low, u, v):
    seed, x, z = rich
    radius = 620
    case = (seed, radius, low, 221, 0, x - u + radius, z - v + radius, 3000)
    total, got = run(core, mode, 0, *case)
    want_total, want = oracle.search(*case)
    assert want["size"][0] >= 49 and ((want["center_x"] == 16 * x + 8) & (want["center_z"] == 16 * z + 8)).any()
    assert total == want_total
    assert np.array_equal(got, want)


# Unions counted by twos and fours at low thresholds: at 28 about a fifth of them reach it.
@pytest.mark.parametrize("mode", [4, 5, 7])
@pytest.mark.parametrize("joined", [1, 2, 4])
@pytest.mark.parametrize("radius", [0, 8, 40, 247, 248, 503, 504, 741])
def test_forced_unions_match_the_oracle(core, oracle, mode, joined, radius):
    rng = np.random.Generator(np.random.PCG64(7000 + 10 * radius + mode + joined))
    for low, high, inner in ((28, 221, 0), (20, 24, 0), (33, 221, radius // 2), (0, 221, 0)):
        if low == 0 and radius > 100:
            continue
        seed = int(rng.integers(-(2**63), 2**63, dtype=np.int64))
        cx, cz = (int(v) for v in rng.integers(-1_800_000, 1_800_001, 2))
        case = (seed, radius, low, high, inner, cx, cz, 3000)
        total, got = run(core, mode, joined, *case)
        want_total, want = oracle.search(*case)
        assert total == want_total
        assert np.array_equal(got, want)


@pytest.mark.parametrize("radius", [80_000, 140_000, 200_000, 270_000])
def test_every_mode_finds_the_same_sites(core, radius):
    """Groups of copies, independent bands, columns in words and the shared LCG against the general scan."""
    case = (4242, radius, 50, 221, 0, -31_337, 65_537, 2000)
    want = run(core, 1, 0, *case)
    for mode in (2, 3, 4, 5, 6, 7):
        got = run(core, mode, 0, *case)
        assert got[0] == want[0], mode
        assert np.array_equal(got[1], want[1]), mode


def test_batch_and_server_use_the_same_unions(core, oracle):
    from slime_b200.lib import SlimeServer
    from slime_b200.workloads import Search
    qs = [Search(seed=s, center_x=10 * s, center_z=-s, radius=300 + s, min_size=30, max_results=500) for s in range(1, 7)]
    wants = [oracle.search(q.seed, q.radius, 30, 221, 0, q.center_x, q.center_z, 500) for q in qs]
    core.lib.slime_b200_set_engine(5, 0)
    try:
        for joined in (1, 2, 4):
            core.lib.slime_b200_set_plane_union(joined)
            for (t, r), (wt, wr) in zip(core.search_batch(qs), wants):
                assert t == wt and np.array_equal(r, wr)
            with SlimeServer(core=core) as server:
                tickets = [server.submit(q) for q in qs]
                for ticket, (wt, wr) in zip(tickets, wants):
                    assert server.wait(ticket) == server.DONE
                    t, r, _ = server.take(ticket, 500)
                    assert t == wt and np.array_equal(r, wr)
    finally:
        core.lib.slime_b200_set_engine(0, 0)
        core.lib.slime_b200_set_plane_union(0)


def test_other_numbers_are_refused(core):
    for joined in (3, 5, 8, -1):
        assert core.lib.slime_b200_set_plane_union(joined) == -1
    assert core.lib.slime_b200_set_plane_union(2) == 0
    assert core.lib.slime_b200_set_plane_union(0) == 2
