import os
import sys
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parent.parent
if str(ROOT) not in sys.path:
    sys.path.insert(0, str(ROOT))


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (B200, sm_100a)")
    config.addinivalue_line("markers", "slow: longer CPU test")


def _skip_without_reference(outcome):
    # A test that needs the reference's own code is skipped where its sources
    # are absent (have_ref), instead of failing for a library that cannot be built.
    if outcome.excinfo is not None:
        import oracle
        if isinstance(outcome.excinfo[1], oracle.ReferenceNotBuilt):
            outcome.force_exception(pytest.skip.Exception("oracle/_ref not built", _use_item_location=True))


@pytest.hookimpl(hookwrapper=True)
def pytest_runtest_setup(item):
    _skip_without_reference((yield))


@pytest.hookimpl(hookwrapper=True)
def pytest_runtest_call(item):
    _skip_without_reference((yield))


@pytest.fixture(scope="session")
def rb():
    import renderbox2_b200
    renderbox2_b200.lib()  # fails loudly if librb2.so is missing
    return renderbox2_b200


@pytest.fixture(scope="session")
def orc():
    import oracle
    return oracle


@pytest.fixture(scope="session")
def cuda():
    import torch
    if not torch.cuda.is_available():
        pytest.fail("CUDA device required for -m gpu tests")
    torch.cuda.init()
    return torch
