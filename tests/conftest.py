"""Shared pytest configuration: the ``gpu`` marker and import paths."""
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
if str(ROOT) not in sys.path:
    sys.path.insert(0, str(ROOT))

GOLDEN = ROOT / "tests" / "golden"


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (run on the B200 box)")


@pytest.fixture(scope="session")
def golden():
    import numpy as np

    def load(name):
        return np.load(GOLDEN / name)

    return load


@pytest.fixture
def new_stream():
    """Makes streams that have run nothing, and so have no scratch: torch hands out 32 in turn."""
    import torch
    from cuda.bindings import runtime

    def make():
        err, handle = runtime.cudaStreamCreateWithFlags(runtime.cudaStreamNonBlocking)
        assert int(err) == 0
        stream = torch.cuda.ExternalStream(int(handle))      # (never destroyed: its handle does not come back)
        stream.wait_stream(torch.cuda.current_stream())
        return stream

    return make
