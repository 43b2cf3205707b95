import os
import sys

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
for p in (REPO, os.path.join(REPO, "luminis-mc_b200")):
    if p not in sys.path:
        sys.path.insert(0, p)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA GPU (B200, sm_100a)")
    config.addinivalue_line("markers", "reference: needs the reference built under oracle/_ref")


def pytest_collection_modifyitems(items):
    """test_gpu_refbind runs the reference's own objects: without the reference's module there
    is nothing to run (test_refbind skips in the same case)."""
    if os.path.isdir(os.path.join(REPO, "oracle", "_ref", "pin", "luminis_mc")):
        return
    for item in items:
        if item.path.name == "test_gpu_refbind.py":
            item.add_marker(pytest.mark.skip(reason="the reference is not built under oracle/_ref"))


def gpu_available() -> bool:
    try:
        import torch
        return torch.cuda.is_available()
    except Exception:
        return False


@pytest.fixture(scope="session")
def cuda():
    if not gpu_available():
        pytest.fail("this test needs a CUDA GPU")
    import torch
    return torch.device("cuda:0")
