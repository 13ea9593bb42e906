import os
import sys

import pytest

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (run on a B200 with `-m gpu`)")
    config.addinivalue_line("markers", "slow: long-running CPU test")


def pytest_collection_modifyitems(config, items):
    import torch
    if torch.cuda.is_available():
        return
    skip = pytest.mark.skip(reason="no CUDA device")
    for item in items:
        if "gpu" in item.keywords:
            item.add_marker(skip)


@pytest.fixture(autouse=True)
def embedding_switch_as_found():
    """`set_deterministic(False)` also selects the float atomics of the embedding gradient, which the tests that follow must not
    inherit: training runs that are compared with one another would differ in the last bits."""
    native = sys.modules.get("superscaler_b200.ops.native")
    ext = getattr(native, "_mod", None)
    before = ext.embedding_in_order() if ext is not None else None
    yield
    if before is not None:
        ext.set_embedding_in_order(before)
