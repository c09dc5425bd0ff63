"""Biome-filtered searches whose emission gate lies above the threshold and whose best sites nearly all
fail the filter. Band searches send the sites from the gate on, and every site in range whose window
holds a redrawn chunk whatever its count: one of those below the gate must not take the place of sites
that were not sent. The world seeds put a redrawn slime chunk at the edge of a Deep Dark region (large
biomes) that covers the rest of the area. The check ranks and filters every centre of the area."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

RADIUS = 60
# Seed, centre; the redrawn chunk lies 50 chunks away from the centre on one or both axes.
AREAS = [(8695192817322579467, 191849, 153809), (-7011834758976442933, -105811, -191186),
         (-2205439178549446247, -103597, 68992)]
FLAGS = 1 | 4  # Deep Dark, large biomes


@pytest.fixture(scope="module")
def core():
    from slime_b200.lib import SlimeCoreB200
    return SlimeCoreB200()


@pytest.fixture(scope="module")
def passing():
    """Per area: the sites that pass, in rank order."""
    from oracle.oracle import BiomeOracle, Oracle
    oracle, biomes, out = Oracle(), BiomeOracle(), {}
    for seed, cx, cz in AREAS:
        n = 2 * RADIUS + 1
        count = oracle.window_counts(seed, cx - RADIUS, cz - RADIUS, n, n).ravel()
        z, x = (v.ravel() for v in np.mgrid[cz - RADIUS:cz + RADIUS + 1, cx - RADIUS:cx + RADIUS + 1])
        keep = (biomes.filter(2602, seed, x, z, 1, 1) & 1) == 0
        order = np.lexsort((z, x, -count))
        order = order[keep[order]]
        out[seed] = np.stack([count[order], 16 * x[order] + 8, 16 * z[order] + 8], axis=1)
    return out


def columns(records):
    return np.stack([records[f] for f in ("size", "center_x", "center_z")], axis=1)


@pytest.mark.parametrize("area", AREAS)
@pytest.mark.parametrize("top", [1, 20, 80, 120, 300])
@pytest.mark.parametrize("mode", [4, 5, 7])
def test_sites_below_the_gate_do_not_rank(core, passing, area, top, mode):
    seed, cx, cz = area
    core.lib.slime_b200_set_engine(mode, 0)
    try:
        total, got = core.search_biome(seed, RADIUS, 0, 221, 0, cx, cz, top, 0, FLAGS, 2602)
    finally:
        core.lib.slime_b200_set_engine(0, 0)
    assert core.lib.slime_b200_last_rare_chunks() > 0
    assert total == (2 * RADIUS + 1) ** 2
    assert np.array_equal(columns(got), passing[seed][:top])


@pytest.mark.parametrize("top", [20, 80, 300])
def test_served_sites_below_the_gate_do_not_rank(core, passing, top):
    from slime_b200.lib import SlimeServer
    from slime_b200.workloads import Search
    core.lib.slime_b200_set_engine(5, 0)
    try:
        with SlimeServer(core=core) as server:
            tickets = [server.submit(Search(seed=seed, center_x=cx, center_z=cz, radius=RADIUS, min_size=0,
                                            max_results=top, biome_flags=FLAGS)) for seed, cx, cz in AREAS]
            for ticket, (seed, _, _) in zip(tickets, AREAS):
                assert server.wait(ticket) == server.DONE
                total, got, _ = server.take(ticket, top)
                assert total == (2 * RADIUS + 1) ** 2
                assert np.array_equal(columns(got), passing[seed][:top])
    finally:
        core.lib.slime_b200_set_engine(0, 0)
