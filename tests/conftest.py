import os
import sys

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)

GOLDEN = os.path.join(ROOT, "tests", "golden")


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (B200); parity tests through the C ABI")


def _skip_without_reference(outcome):
    """A test or fixture that asks for the reference oracle where it cannot be built is skipped."""
    import oracle

    e = outcome.excinfo[1] if outcome.excinfo else None
    if isinstance(e, oracle.ReferenceMissing):
        outcome.force_exception(pytest.skip.Exception("reference oracle library not built (oracle/_ref)"))


@pytest.hookimpl(hookwrapper=True)
def pytest_runtest_setup(item):
    _skip_without_reference((yield))


@pytest.hookimpl(hookwrapper=True)
def pytest_runtest_call(item):
    _skip_without_reference((yield))


@pytest.fixture(scope="session")
def golden():
    def load(name):
        return np.load(os.path.join(GOLDEN, name))
    return load
