import os
import sys
from pathlib import Path

# One BLAS code path on every x86 host, set before torch is first imported: the oracle's pinned outputs were made on another
# CPU model, and some models' default fp32 summation order moves single bf16 roundings, which the recurrence carries on to
# the following rows. Here and not in the oracle, which the benchmark times: it takes MKL two to five times longer.
os.environ.setdefault("MKL_CBWR", "COMPATIBLE")

import pytest

ROOT = Path(__file__).resolve().parent.parent
if str(ROOT) not in sys.path:
    sys.path.insert(0, str(ROOT))


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (run on the B200 box)")


def pytest_collection_modifyitems(config, items):
    import torch

    if torch.cuda.is_available():
        return
    skip = pytest.mark.skip(reason="no CUDA device")
    for item in items:
        if "gpu" in item.keywords:
            item.add_marker(skip)


@pytest.fixture(scope="session")
def lib():
    from tensorfold_b200 import _lib, build

    build.build()
    return _lib.load()
