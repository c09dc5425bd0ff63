import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
if str(ROOT) not in sys.path:
    sys.path.insert(0, str(ROOT))


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (run with -m gpu)")


@pytest.hookimpl(wrapper=True)
def pytest_runtest_call(item):
    """A test that comes to a reference library which is not built here is reported as skipped there, with
    the library's name; what it checked before that has been checked."""
    from oracle.oracle import ReferenceNotBuilt
    try:
        return (yield)
    except ReferenceNotBuilt as e:
        pytest.skip(str(e))


@pytest.fixture(scope="session")
def oracle():
    from oracle.oracle import Oracle
    return Oracle()


@pytest.fixture(scope="session")
def golden():
    import numpy as np
    d = ROOT / "tests" / "golden"
    return {name: np.load(d / f"{name}.npz") for name in ("predicate", "search", "precise")}
