"""Searches that other tests compare with the reference's libraries, against this repository's oracle: those
libraries can only be built where the reference's source tree is. Annuli in every mode, and requests of a
batch and of the server with their precise scores."""
import numpy as np
import pytest

from slime_b200.workloads import Search

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def core():
    from slime_b200.lib import SlimeCoreB200
    core = SlimeCoreB200()
    core.set_y_scan_config(0, -64, -64, 64, 4)
    return core


def check(oracle, q, total, res):
    want_total, want = oracle.search(q.seed, q.radius, q.min_size, q.max_size, q.rd_min, q.center_x, q.center_z,
                                     q.max_results, q.precise_afk, precise_limit=100)
    assert total == want_total, q
    assert np.array_equal(res, want), q


@pytest.mark.parametrize("mode", [0, 1, 2, 3, 4, 5, 6, 7])
@pytest.mark.parametrize("q", [
    Search(2718281828, 250_000, -90_000, 20_000, 40, rd_min=18_000, max_results=3000),
    Search(-161803, -1_000_000, 1_000_000, 6_000, 38, max_size=45, rd_min=5_400, max_results=800),
    Search(5, 70_000, 0, 15_000, 36, rd_min=14_990, max_results=5000),
    Search(77, -3, 9, 12_000, 44, rd_min=4_000, max_results=500),
])
def test_annuli(core, oracle, q, mode):
    core.lib.slime_b200_set_engine(mode, 0)
    try:
        total, res = core.search(q.seed, q.radius, q.min_size, q.max_size, q.rd_min, q.center_x, q.center_z, q.max_results)
    finally:
        core.lib.slime_b200_set_engine(0, 0)
    check(oracle, q, total, res)


MIX = [
    Search(11, 0, 0, 300, 30, max_results=5000),
    Search(-12, 500_000, -20, 20_000, 45, max_results=300),
    Search(14, 7, 7, 2_000, 28, max_size=33, max_results=50),
    Search(15, 0, 9_000, 9_000, 40, rd_min=5_000, max_results=700),
    Search(16, 1, 2, 1_500, 20, max_results=100),
    Search(17, 0, 0, 14_000, 46, max_results=150, precise_afk=1),
    Search(18, 0, 0, 100, 60, max_results=10),
    Search(19, -3, 3, 0, 0, max_results=4),
    Search(20, 100, 100, 4_000, 36, max_results=3),
    Search(21, -8, 8, 11_000, 39, rd_min=10_500, max_results=2000),
]


def test_batch(core, oracle):
    for q, (total, res) in zip(MIX, core.search_batch(MIX)):
        check(oracle, q, total, res)


def test_server(core, oracle):
    from slime_b200.lib import SlimeServer
    with SlimeServer(core=core) as server:
        tickets = [server.submit(q) for q in MIX]
        for ticket, q in zip(tickets, MIX):
            assert server.wait(ticket) == server.DONE
            total, res, _ = server.take(ticket, q.max_results)
            check(oracle, q, total, res)


def test_biome_search_scores(core, oracle):
    """Precise scores of a biome-filtered search are those of the sites by themselves."""
    for seed in (3, 4):
        total, plain = core.search_biome(seed, 3000, 40, 221, 0, 50_000, -50_000, 60, 0, 3, 2602)
        total2, scored = core.search_biome(seed, 3000, 40, 221, 0, 50_000, -50_000, 60, 1, 3, 2602)
        assert total == total2 and len(plain)
        assert np.array_equal(scored, oracle.score_precise(seed, plain, 1))
