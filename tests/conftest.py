import importlib
import os
import sys

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)
ORACLE_DIR = os.path.join(ROOT, "oracle")
if ORACLE_DIR not in sys.path:
    sys.path.insert(0, ORACLE_DIR)

GOLDEN = os.path.join(ROOT, "tests", "golden", "golden.npz")


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA GPU (B200, sm_100a)")


REFERENCE = os.path.join(ORACLE_DIR, "_ref", "libgirref.so")
NEED_REFERENCE = ("test_incremental_matches_reference_and_scratch", "test_reachable_matches_reference",
                  "test_betweenness_matches_reference")


def pytest_collection_modifyitems(items):
    """Where the compiled reference is missing, the tests that cannot do without it run (and fail) behind the others, so
    that a run that stops at the first failure gets to those; test_zz_no_alloc.py stays last."""
    if not os.path.exists(REFERENCE):
        items.sort(key=lambda i: (i.path.name == "test_zz_no_alloc.py",
                                  getattr(i, "originalname", i.name) in NEED_REFERENCE))


@pytest.fixture(scope="session")
def pkg():
    return importlib.import_module("graph-intermedia-representation_b200")


@pytest.fixture(scope="session")
def orc():
    import oracle
    oracle.lib()
    return oracle


@pytest.fixture(scope="session")
def golden():
    return dict(np.load(GOLDEN))


def golden_cases(g):
    return [str(x) for x in g["cases"]]
