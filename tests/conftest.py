import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (run with -m gpu on a B200)")


@pytest.fixture(autouse=True)
def _default_settings(request):
    """The library's launch settings are process-wide: every GPU test starts from the defaults, whatever the one before set."""
    if "gpu" in request.keywords:
        from adamas_b200 import _kernels as K
        K.set_max_cluster(int(os.environ.get("ADAMAS_MAX_CLUSTER", 8)))
        K.set_estimate_blocks_per_sm(int(os.environ.get("ADAMAS_EST_BLOCKS_PER_SM", 2)))
        K.set_fused_append(os.environ.get("ADAMAS_FUSED_APPEND", "1") != "0")


def pytest_collection_modifyitems(config, items):
    import torch
    if torch.cuda.is_available():
        return
    skip = pytest.mark.skip(reason="no CUDA device")
    for item in items:
        if "gpu" in item.keywords:
            item.add_marker(skip)
