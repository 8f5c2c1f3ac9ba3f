import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (run on a B200)")


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


GOLDEN = os.path.join(ROOT, "tests", "golden")


@pytest.fixture
def golden():
    import numpy as np

    def load(name):
        with np.load(os.path.join(GOLDEN, name + ".npz")) as z:
            return {k: z[k] for k in z.files}
    return load


@pytest.fixture(autouse=True)
def pruned_form_at_every_size(request, monkeypatch):
    """The tests of the pruned form use shapes at its edges, below the sizes from which the wrappers ask for it."""
    if request.module.__name__ == "test_prune_gpu":
        from sortnet_b200 import norm_dist_cuda
        monkeypatch.setattr(norm_dist_cuda, "_prune_pays", lambda *sizes: True)
