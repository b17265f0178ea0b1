import os
import sys

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "sph-erosion_gb300")
ORACLE = os.path.join(ROOT, "oracle")
GOLDEN = os.path.join(ROOT, "tests", "golden")
for p in (PKG, ORACLE, ROOT):
    if p not in sys.path:
        sys.path.insert(0, p)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA GPU (runs the sm_103a kernels)")


def pytest_collection_modifyitems(items):
    """The one test that runs the reference's own code needs its sources: an
    empty reference directory counts as none."""
    if not os.path.isfile("/root/reference/Erosion/fluid_system.h"):
        for item in items:
            if item.name == "test_reference_harness_matches_when_present":
                item.add_marker(pytest.mark.skip(reason="reference sources absent"))


@pytest.fixture(scope="session")
def golden():
    cache = {}

    def load(name):
        if name not in cache:
            with np.load(os.path.join(GOLDEN, name)) as z:
                cache[name] = {k: z[k] for k in z.files}
        return cache[name]

    return load


@pytest.fixture(scope="session")
def oracle_lib():
    import oracle as O

    O.build()
    return O
