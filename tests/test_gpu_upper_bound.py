"""Upper bounds above the 221 cells of a window mean no bound, in every entry point: the argument checks
take any max_size >= min_size, and the count histograms end at 221."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SEED, RADIUS, LOW, CX, CZ, TOP = 4711, 300, 33, 70_000, -5_000, 400


@pytest.fixture(scope="module")
def core():
    from slime_b200.lib import SlimeCoreB200
    return SlimeCoreB200()


@pytest.fixture(scope="module")
def want(oracle):
    return oracle.search(SEED, RADIUS, LOW, 221, 0, CX, CZ, TOP)


@pytest.mark.parametrize("high", [222, 256, 2**31 - 1])
@pytest.mark.parametrize("mode", [0, 2, 3, 4, 5, 6, 7])
def test_search(core, want, mode, high):
    core.lib.slime_b200_set_engine(mode, 0)
    try:
        total, got = core.search(SEED, RADIUS, LOW, high, 0, CX, CZ, TOP)
    finally:
        core.lib.slime_b200_set_engine(0, 0)
    assert total == want[0]
    assert np.array_equal(got, want[1])


@pytest.mark.parametrize("high", [222, 2**31 - 1])
def test_other_entry_points(core, want, high):
    from slime_b200.lib import RESULT_DTYPE, SlimeServer
    from slime_b200.workloads import Search
    q = Search(seed=SEED, center_x=CX, center_z=CZ, radius=RADIUS, min_size=LOW, max_size=high, max_results=TOP)
    band = Search(seed=SEED, center_x=CX, center_z=CZ, radius=RADIUS, min_size=44, max_size=high, max_results=TOP)
    (total, got), (few, _) = core.search_batch([q, band])
    assert total == want[0] and np.array_equal(got, want[1])
    assert few == int((want[1]["size"] >= 44).sum())
    with SlimeServer(core=core) as server:
        ticket = server.submit(q)
        assert server.wait(ticket) == server.DONE
        total, got, _ = server.take(ticket, TOP)
        assert total == want[0] and np.array_equal(got, want[1])
    buf = np.zeros(TOP, dtype=RESULT_DTYPE)
    total = core.lib.slime_b200_search_noalloc(SEED, RADIUS, LOW, high, 0, CX, CZ,
                                               buf.ctypes.data_as(ctypes.c_void_p), TOP)
    assert total == want[0] and np.array_equal(buf[:len(want[1])], want[1])
