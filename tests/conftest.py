import os
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
if ROOT not in sys.path:
    sys.path.insert(0, ROOT)


def pytest_configure(config):
    config.addinivalue_line("markers", "gpu: needs a CUDA GPU (B200); runs through libmdb200.so")


def pytest_collection_modifyitems(config, items):
    """The tests that run the reference's own kernels need them built, or the
    reference's sources to build them from."""
    from oracle import build_ref, refkernels

    source = os.path.join(build_ref.reference_tree(), "src", "md_cuda_common.cu")
    if refkernels.available() or os.path.exists(source):
        return
    skip = pytest.mark.skip(reason="the reference's kernels are not built and its sources are "
                                   "not here (oracle/build_ref.py)")
    for item in items:
        if item.path.name == "test_gpu_ref_kernels.py":
            item.add_marker(skip)


@pytest.fixture(scope="session")
def built():
    """Builds the library and the oracle once per session."""
    import __graft_entry__

    __graft_entry__.build()
    return True
