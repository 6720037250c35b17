import functools
import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (B200); run with -m gpu")


def pytest_collection_modifyitems(config, items):
    import torch
    if torch.cuda.is_available():
        return
    skip = pytest.mark.skip(reason="no CUDA device")
    for item in items:
        if "gpu" in item.keywords:
            item.add_marker(skip)


@pytest.fixture(autouse=True)
def results_of_ranks_by_value(request, monkeypatch):
    """The gloo ranks may be gone before the test has read what they sent (see helpers.run_rank)."""
    if request.module.__name__ != "test_ep_gloo":
        return
    import helpers
    for worker in ("_worker", "_leaver_worker"):
        monkeypatch.setattr(request.module, worker, functools.partial(helpers.run_rank, "test_ep_gloo", worker))
