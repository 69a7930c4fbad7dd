import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (run with -m gpu on a B200)")


@pytest.fixture(scope="session")
def port_lib():
    from oracle import pyoracle
    pyoracle.build("port")
    return pyoracle


@pytest.hookimpl(hookwrapper=True)
def pytest_runtest_call(item):
    """A test that needs a checker compiled from the SNAC tree is skipped where neither is there."""
    from oracle.pyoracle import CheckerMissing
    outcome = yield
    if outcome.excinfo and issubclass(outcome.excinfo[0], CheckerMissing):
        outcome.force_exception(pytest.skip.Exception(str(outcome.excinfo[1])))
