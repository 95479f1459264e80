import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA GPU (B200) and the built libxsolver_b200.so")


def gpu_available():
    try:
        import torch

        return torch.cuda.is_available()
    except Exception:
        return False


@pytest.fixture(autouse=True)
def schedule_defaults(request):
    """The options of the exact solves' schedules are process-wide, and some
    (a box size, the lines' row limits) have no setter that undoes them:
    every GPU test ends with all of them at their defaults."""
    yield
    if "cuda" in request.fixturenames:
        from xsolver_b200 import _lib

        assert _lib.lib().xs_reset_trsv_tuning() == 0


@pytest.fixture(scope="session")
def cuda():
    if not gpu_available():
        pytest.fail("GPU test selected but no CUDA device is visible")
    import torch

    return torch.device("cuda:0")
