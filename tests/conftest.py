import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA GPU (B200) and librpb200.so")


def pytest_collection_modifyitems(items):
    # Where the reference's own code could not be built (its checkout is absent) the
    # tests of that build fail: last, so that a run that ends at the first failure
    # has run the others.
    if not os.path.exists(os.path.join(ROOT, "oracle", "_ref", "dropin_driver")):
        items.sort(key=lambda item: item.path.name == "test_gpu_dropin.py")


@pytest.fixture(scope="session")
def cuda():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import reapers_b200 as rb
    rb.init(0)
    return torch.device("cuda:0")
