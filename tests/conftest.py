import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (B200, sm_100a)")


def cuda_available():
    try:
        import torch
        return torch.cuda.is_available()
    except Exception:
        return False


# tests that assert the reference's own build (oracle/_ref): last where it is
# absent, so that a run which stops at the first failure gets to all the others
NEEDS_REFERENCE = ("test_fp32_unit_vs_reference",)


def pytest_collection_modifyitems(config, items):
    from oracle import oracle as O

    if not O.have_ref():
        items.sort(key=lambda it: getattr(it, "originalname", it.name) in NEEDS_REFERENCE)
    if cuda_available():
        return
    skip = pytest.mark.skip(reason="no CUDA device")
    for it in items:
        if "gpu" in it.keywords:
            it.add_marker(skip)
