"""pytest configuration: the ``gpu`` marker and import paths.

Tests marked ``gpu`` need a B200 and call the CUDA library through its C ABI;
everything else (oracle vs golden vectors, host-side validation, exported
symbols) runs on CPU.
"""
import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
for p in (ROOT, os.path.join(ROOT, "mlx-serve_b200")):
    if p not in sys.path:
        sys.path.insert(0, p)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (B200); runs the CUDA kernels through the C ABI")


def _has_gpu():
    try:
        import torch

        return torch.cuda.is_available()
    except Exception:
        return False


def pytest_collection_modifyitems(config, items):
    if _has_gpu():
        return
    skip = pytest.mark.skip(reason="no CUDA device")
    for item in items:
        if "gpu" in item.keywords:
            item.add_marker(skip)


@pytest.fixture
def no_clusters():
    import qb200
    qb200.lib().qb200_debug_refuse_clusters(True)
    yield
    qb200.lib().qb200_debug_refuse_clusters(False)
