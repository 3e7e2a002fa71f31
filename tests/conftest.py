import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
for p in (os.path.join(ROOT, "pbe-fixed-pivot-cuda_gb300"), os.path.join(ROOT, "oracle"), ROOT):
    if p not in sys.path:
        sys.path.insert(0, p)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA GPU (sm_103a)")


@pytest.fixture(scope="session", autouse=True)
def _built():
    """Make sure the library and the oracle are built (incremental, seconds)."""
    import __graft_entry__

    __graft_entry__.build()
    yield


def pytest_collection_modifyitems(config, items):
    try:
        import torch

        has_gpu = torch.cuda.is_available()
    except Exception:  # pragma: no cover
        has_gpu = False
    # tests that need the reference's sources staged under oracle/_ref fail where they are
    # not: last, so that a run that stops at the first failure has been through the others
    if not os.path.isdir(os.path.join(ROOT, "oracle", "_ref", "examples")):
        items.sort(key=lambda item: "example_bins" in getattr(item, "fixturenames", ()))
    if has_gpu:
        return
    skip = pytest.mark.skip(reason="no CUDA device in this environment")
    for item in items:
        if "gpu" in item.keywords:
            item.add_marker(skip)
