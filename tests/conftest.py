import gc
import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (run with -m gpu on a B200)")


@pytest.fixture(scope="session")
def oracle():
    from oracle import api
    api.build()
    return api


@pytest.fixture(scope="session")
def lib():
    """The loaded C-ABI library; GPU tests fail (not skip) when it is missing."""
    from helix_b200 import _lib
    return _lib.load()


@pytest.fixture(autouse=True)
def collect_garbage_before_allocation_counts(request):
    """Exceptions kept by earlier tests hold their frames' tensors in reference cycles; a collection in the middle of a test
    that compares allocator counters would look like an allocation of its own."""
    if "no_alloc" in request.module.__name__:
        gc.collect()
    yield
