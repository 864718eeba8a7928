import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
for sub in ("solveit-code_gb300", "oracle", "tests"):
    p = os.path.join(ROOT, sub)
    if p not in sys.path:
        sys.path.insert(0, p)

# an empty reference directory is no reference tree
_ref = os.environ.get("SOLVEIT_REFERENCE", "/root/reference")
if os.path.isdir(_ref) and not os.listdir(_ref):
    os.environ["SOLVEIT_REFERENCE"] = os.path.join(_ref, "absent")


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA GPU (GB300, sm_103a)")


GOLDEN = os.path.join(ROOT, "tests", "golden")


@pytest.fixture(scope="session")
def golden_dir():
    return GOLDEN
