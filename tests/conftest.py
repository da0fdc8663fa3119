import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (B200)")


def cuda_available():
    try:
        import torch
        return torch.cuda.is_available()
    except Exception:
        return False


def pytest_collection_modifyitems(config, items):
    if cuda_available():
        return
    skip = pytest.mark.skip(reason="no CUDA device")
    for item in items:
        if "gpu" in item.keywords:
            item.add_marker(skip)


def _reference_missing(e):
    """A test that stopped because the reference's own build is not there (it is made
    from the reference's source tree, which is not part of this repository)."""
    from oracle import refbind
    return (isinstance(e, OSError) and not refbind.have_host() and
            "oracle/_ref/" in str(e).replace(os.sep, "/"))


@pytest.hookimpl(wrapper=True)
def pytest_runtest_setup(item):
    try:
        return (yield)
    except OSError as e:
        if _reference_missing(e):
            pytest.skip("reference build missing (make -C oracle ref)")
        raise


@pytest.hookimpl(wrapper=True)
def pytest_runtest_call(item):
    try:
        return (yield)
    except OSError as e:
        if _reference_missing(e):
            pytest.skip("reference build missing (make -C oracle ref)")
        raise


@pytest.fixture(scope="session")
def ref_host():
    from oracle import refbind
    path = os.path.join(refbind.REF_DIR, "libawpref_host.so")
    if not os.path.exists(path):
        pytest.skip("reference host build missing (make -C oracle ref)")
    return refbind.RefHost()
