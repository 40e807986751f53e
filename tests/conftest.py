import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (B200)")


def has_gpu():
    try:
        import torch
        return torch.cuda.is_available()
    except Exception:
        return False


def pytest_collection_modifyitems(config, items):
    if has_gpu():
        return
    skip = pytest.mark.skip(reason="no CUDA device")
    for it in items:
        if "gpu" in it.keywords:
            it.add_marker(skip)


@pytest.fixture(autouse=True)
def default_switches(request):
    """Every GPU test starts from the library's default switches, whatever an earlier one left."""
    yield
    if "gpu" in request.keywords:
        import fmmlib3d_b200 as F
        F.set_precision(0)
        F.set_precision_thread(-1)
        F.set_m2l_mode(0)
        F.set_tensor_m2l(3)
        F.set_overlap(True)
        F.set_tuning_cache(None)
