"""Without the reference's kernels, and without its sources, the tests that run them
are skipped: they say why, and the ones after them run."""
import os
import subprocess
import sys

import pytest

from oracle import refkernels
from tests.conftest import ROOT


def test_tests_of_the_reference_kernels_are_skipped():
    if refkernels.available():
        pytest.skip("the reference's kernels are built")
    env = dict(os.environ, MDB_REFERENCE_TREE=os.path.join(ROOT, "no-such-tree"))
    r = subprocess.run([sys.executable, "-m", "pytest", "-q", "-x", "-rs", "-p", "no:cacheprovider",
                        os.path.join(ROOT, "tests", "test_gpu_ref_kernels.py")],
                       cwd=ROOT, env=env, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout[-2000:]
    assert "skipped" in r.stdout and "passed" not in r.stdout and "not built" in r.stdout
