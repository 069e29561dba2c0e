import os
import sys

import pytest

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(REPO, "inspire-gpu_b200"))
sys.path.insert(0, os.path.join(REPO, "tests"))


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA GPU (B200, sm_100a)")
    config.addinivalue_line("markers", "slow: long-running case")


def gpu_available():
    try:
        import torch
        return torch.cuda.is_available()
    except Exception:
        return False


# Tests whose child processes use the reference's CPU library.
REF_LIB_CHILDREN = ("test_sharded_gather_reproduces_the_single_process_answer",)


def skip_without_reference_library(items):
    """The reference's own CPU library is built from its sources (oracle/Makefile,
    REF=...).  Where it is not, the tests that use it are skipped, as those of its
    GPU library are; tests against the oracle and the golden files remain."""
    import oracle_lib
    if os.path.exists(oracle_lib.REF_SO):
        return
    reason = "reference CPU library not built (needs the reference sources)"
    oracle_lib.RefLib.__init__ = lambda self, *a: pytest.skip(reason)
    for it in items:
        if getattr(it, "originalname", None) in REF_LIB_CHILDREN:
            it.add_marker(pytest.mark.skip(reason=reason))


def pytest_collection_modifyitems(config, items):
    skip_without_reference_library(items)
    if gpu_available():
        return
    skip = pytest.mark.skip(reason="no CUDA GPU in this container")
    for it in items:
        if "gpu" in it.keywords:
            it.add_marker(skip)


@pytest.fixture(scope="session")
def oracle():
    from oracle_lib import Oracle
    return Oracle()


@pytest.fixture(scope="session")
def ref():
    from oracle_lib import RefLib
    return RefLib()
