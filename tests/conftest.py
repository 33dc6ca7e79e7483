import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (B200, sm_100a)")


@pytest.hookimpl(hookwrapper=True)
def pytest_runtest_call(item):
    """A test that gets as far as a comparison with the reference's own library, which is not built here, is
    reported as skipped with that reason."""
    outcome = yield
    if outcome.excinfo is not None:
        from oracle.ref_sim import NotBuilt

        if issubclass(outcome.excinfo[0], NotBuilt):
            outcome.force_exception(pytest.skip.Exception(str(outcome.excinfo[1])))
