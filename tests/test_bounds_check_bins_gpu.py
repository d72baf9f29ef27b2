"""The two-pass SpMV under the checking build of the library: its own tests pass, and a layout with one bad number is refused
with a record.  The library is chosen when the package is imported, so both run in child processes."""

import os

import pytest

from test_bounds_check_gpu import HERE, _child

pytestmark = pytest.mark.gpu


def test_bad_layouts_are_refused(cuda):
    r = _child([os.path.join(HERE, "bounds_check_bins_cases.py")], 600)
    assert r.returncode == 0, (r.stdout + r.stderr)[-4000:]
    assert "all cases ok" in r.stdout


def test_good_layouts_pass(cuda):
    # (without the call that is recorded in a CUDA graph: the walk reads its record back)
    r = _child(["-m", "pytest", os.path.join(HERE, "test_bins_gpu.py"), "-m", "gpu", "-q", "-x", "-p", "no:cacheprovider", "-k",
                "edges or infinities or empty_rows or over_two_slices or left_to_one_pass"], 900)
    assert r.returncode == 0, (r.stdout + r.stderr)[-4000:]
    assert " passed" in r.stdout and " failed" not in r.stdout
