import gc
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
if str(ROOT) not in sys.path:
    sys.path.insert(0, str(ROOT))


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (run with -m gpu on a B200)")


def pytest_collection_finish(session):
    gc.collect()
    gc.freeze()     # what is loaded by now stays: the collections below look at the tests' own objects only


@pytest.fixture(autouse=True)
def _no_leftover_tensors(request):
    """Tensors that an earlier test left in a reference cycle (pytest.raises keeps frames alive) go before the next GPU
    test starts, not in the middle of one that watches the allocator."""
    if request.node.get_closest_marker("gpu"):
        gc.collect()


@pytest.fixture(scope="session")
def golden_dir():
    return ROOT / "tests" / "golden"
