import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (run on the B200 box)")


@pytest.fixture
def kernel_of():
    """Name of the kernel that a call launched last (which of several a size went to)."""
    def name(call):
        from latentq_llm_b200 import _lib
        call()
        return _lib.lib.lq_last_launch().decode()
    return name


@pytest.fixture(scope="session")
def golden():
    import numpy as np
    return dict(np.load(os.path.join(ROOT, "tests", "golden", "reference_vectors.npz")))
