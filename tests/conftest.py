import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (B200, sm_100a)")


@pytest.fixture(scope="session")
def oracle():
    from oracle import pyoracle
    pyoracle.build()
    return pyoracle


@pytest.fixture(scope="session")
def ctx():
    """One device context for the GPU tests (fails loudly without a GPU)."""
    from radtrancode_b200 import _lib, cirsradg
    _lib.build()
    c = cirsradg.Context(0)
    yield c
    c.close()


@pytest.fixture(autouse=True)
def _form_chosen_by_the_batch(request):
    """A test that uses the shared context leaves it with no tile and no schedule set."""
    yield
    if "ctx" in request.fixturenames:
        c = request.getfixturevalue("ctx")
        c.set_tile(0)
        c.set_schedule(-1, 0)
