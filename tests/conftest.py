import gc
import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (B200); run with -m gpu")


@pytest.fixture(scope="session")
def backend():
    """Initialises the CUDA backend once per test session (GPU tests only)."""
    import kandle_b200
    return kandle_b200.init(0)


@pytest.fixture(scope="session")
def oracle():
    from oracle import oracle as orc
    orc.build()
    return orc


@pytest.fixture
def collected():
    """For tests that account device memory: no garbage of earlier tests is left when they start.  An exception's traceback
    keeps its frames' tensors until the cycle is collected, which may otherwise happen between two readings."""
    gc.collect()
