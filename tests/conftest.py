import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA GPU (B200) and the built libmpm_b200.so")


def pytest_collection_modifyitems(items):
    # the comparison with the reference build fails where that build is not
    # there: last, so that a run that stops at the first failure has run the rest
    from oracle import ref
    if not ref.available():
        items.sort(key=lambda i: i.path.name == "test_config_parity.py")


def _has_gpu() -> bool:
    try:
        import torch
        return torch.cuda.is_available()
    except Exception:
        return False


@pytest.fixture(scope="session")
def gpu():
    if not _has_gpu():
        pytest.fail("this test needs a GPU; run it with -m gpu on a GPU box")
    from mpm_cuda_b200 import _lib
    return _lib.load()
