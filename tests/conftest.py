import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "lattice-boltzmann-method_b200")
GOLDEN = os.path.join(ROOT, "tests", "golden")
for p in (ROOT, PKG):
    if p not in sys.path:
        sys.path.insert(0, p)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA GPU (B200, sm_100a)")


@pytest.hookimpl(wrapper=True)
def pytest_runtest_call(item):
    """A test that drives the reference's own solver is skipped where that library was not built."""
    from oracle.refmc import ReferenceMissing
    try:
        return (yield)
    except ReferenceMissing as exc:
        pytest.skip(str(exc))


def gpu_available():
    try:
        import torch
        return torch.cuda.is_available()
    except Exception:
        return False


@pytest.fixture(scope="session")
def golden_dir():
    return GOLDEN
