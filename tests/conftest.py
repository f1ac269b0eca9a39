import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA GPU (B200); run with -m gpu")
    config.addinivalue_line("markers", "slow: long-running (large state)")


def _has_gpu() -> bool:
    """A CUDA device is visible (driver API, without importing torch)."""
    import ctypes

    try:
        cuda = ctypes.CDLL("libcuda.so.1")
        if cuda.cuInit(0) != 0:
            return False
        n = ctypes.c_int(0)
        return cuda.cuDeviceGetCount(ctypes.byref(n)) == 0 and n.value > 0
    except OSError:
        return False


HAS_GPU = _has_gpu()


def pytest_collection_modifyitems(config, items):
    # The drop-in tests fail where their programs are not built (they need the
    # reference's sources): a run that stops at its first failure has all the
    # others behind it by then.
    if not os.path.isdir(os.path.join(ROOT, "tests", "dropin", "_build", "bin")):
        items.sort(key=lambda item: item.path.name == "test_gpu_dropin.py")
    if HAS_GPU:
        return
    skip = pytest.mark.skip(reason="no CUDA device in this environment")
    for item in items:
        if "gpu" in item.keywords:
            item.add_marker(skip)
