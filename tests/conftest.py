import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (run with -m gpu on a B200)")


@pytest.fixture(params=["staged", "whole-step"])
def route(request, monkeypatch):
    """The two routes of a matrix that the staged kernels take in large sets and the whole-step kernel in small ones: the
    line between them is moved below or above every set of the test (a plan reads it when it is sized and created)."""
    monkeypatch.setenv("CAME_B200_SMALL_SET_ELEMS", "0" if request.param == "staged" else "1e18")
    return request.param


@pytest.fixture
def staged(monkeypatch):
    monkeypatch.setenv("CAME_B200_SMALL_SET_ELEMS", "0")


def pytest_collection_modifyitems(config, items):
    try:
        import torch
        has_gpu = torch.cuda.is_available()
    except Exception:
        has_gpu = False
    if has_gpu:
        return
    skip = pytest.mark.skip(reason="no CUDA device")
    for item in items:
        if "gpu" in item.keywords:
            item.add_marker(skip)
