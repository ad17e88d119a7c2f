import os
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
for p in (ROOT, os.path.join(ROOT, "tests")):
    if p not in sys.path:
        sys.path.insert(0, p)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA device (B200) and the built library")


def _ensure_oracle():
    lib = os.path.join(ROOT, "oracle", "_ref", "liboracle.so")
    if not os.path.exists(lib):
        subprocess.run(["make", "-C", os.path.join(ROOT, "oracle"), "oracle"], check=True, capture_output=True)


@pytest.fixture(scope="session")
def oracle_lib():
    _ensure_oracle()
    from oracle import orc
    return orc.lib()


def _ref_built():
    d = os.path.join(ROOT, "oracle", "_ref")
    return all(os.path.exists(os.path.join(d, f)) for f in ("libmxshim.so", "libref_mc.so", "libref_heat.so"))


@pytest.fixture(scope="session")
def ref_available():
    """The reference build (oracle/_ref/libref_*.so) exists (built where the reference sources are)."""
    return _ref_built()


# Tests that time the reference itself and do not ask ref_available: they run where it is built.
NEEDS_REF = ("test_reference_arm_prints_one_contract_line",)


def pytest_collection_modifyitems(items):
    if not _ref_built():
        for item in items:
            if item.name in NEEDS_REF:
                item.add_marker(pytest.mark.skip(reason="reference build not available"))
