import os
import sys

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
GOLDEN = os.path.join(ROOT, "tests", "golden")
for p in (ROOT, os.path.join(ROOT, "oracle"), GOLDEN):
    if p not in sys.path:
        sys.path.insert(0, p)


# The adapter tests run where the reference tree is present; an empty mount
# point is not a tree.
if "QCMG_REFERENCE_DIR" not in os.environ and not os.path.isfile("/root/reference/src_qcm/CPT.cpp"):
    os.environ["QCMG_REFERENCE_DIR"] = os.path.join(ROOT, "oracle", "no_reference")


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA GPU (GB300) and the built libqcmg")


def load_golden(name):
    return dict(np.load(os.path.join(GOLDEN, name + ".npz")))


@pytest.fixture
def golden():
    return load_golden
