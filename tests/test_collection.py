"""Tests of the reference's own sources need a binary built from them; where it
is not built they are skipped, so that a run with -x reaches the tests behind
them."""
import os
import subprocess
import sys

import pytest

from oracle import oracle as O

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.skipif(os.path.exists(O.REF_ON_MDF), reason="the reference is built here")
def test_tests_of_the_reference_are_skipped_where_it_is_not_built():
    r = subprocess.run([sys.executable, "-m", "pytest", os.path.join("tests", "test_reference_binding.py"), "-x", "-q",
                        "-p", "no:cacheprovider"], cwd=ROOT, capture_output=True, text=True)
    assert r.returncode == 0 and "5 skipped" in r.stdout and "failed" not in r.stdout, r.stdout
