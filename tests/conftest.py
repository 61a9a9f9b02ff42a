"""Shared fixtures.  GPU tests carry @pytest.mark.gpu; everything else runs on CPU."""
from __future__ import annotations

import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
if str(ROOT) not in sys.path:
    sys.path.insert(0, str(ROOT))

import __graft_entry__ as entry  # noqa: E402


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA GPU (runs the CUDA kernels)")


# Need what is built from the reference's checkout and fail where it is absent: a run that stops at the
# first failure has then run everything else.
REFERENCE_FILES = {"test_gpu_ref_drivers.py", "test_gpu_reference_kernels.py", "test_gpu_reference_speed.py"}


def pytest_collection_modifyitems(items):
    items.sort(key=lambda item: item.path.name in REFERENCE_FILES)


@pytest.fixture(scope="session")
def built():
    entry.build()
    return True


@pytest.fixture(scope="session")
def pkg(built):
    return entry.load_package()


@pytest.fixture(scope="session")
def orc(built):
    return entry.load_oracle()


@pytest.fixture(scope="session")
def cuda(pkg):
    import torch
    if not torch.cuda.is_available():
        pytest.fail("GPU test collected on a machine without CUDA")
    return torch.device("cuda:0")
