"""The bounds-checked build at the edges of the on-chip searches: the tests of
the per-lane bitmaps, the backward search and the wide hand-offs run once
against it, and must pass unchanged.  Every append to a hand-off list is
checked against the list's length."""
import glob
import os
import re
import subprocess
import sys

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
PKG = os.path.join(ROOT, "gpgpu-binary-automaton-synchronizing-algorithms_b200")
CHECKED = os.path.join(PKG, "sbfs", "_lib", "libsbfs_checked.so")
FILES = ["test_lane_bitmaps.py", "test_lane_large_ranks.py", "test_inverse_search.py", "test_device_memory.py",
         "test_n17_launches.py", "test_small_n_counts.py"]


def test_no_unchecked_append():
    for path in glob.glob(os.path.join(PKG, "csrc", "*.cu")):
        text = open(path).read()
        assert not re.search(r"(heavy|left)[_.]list\[\s*(atomicAdd|pos\s*\+)", text), path


@pytest.mark.gpu
def test_edges_under_the_checked_build():
    import torch
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    assert os.path.exists(CHECKED), "build with __graft_entry__.build() first"
    r = subprocess.run([sys.executable, "-m", "pytest", *[os.path.join(ROOT, "tests", f) for f in FILES], "-q", "-m",
                        "gpu", "-k", "not cost and not little_device_memory", "-p", "no:cacheprovider"],
                       env=dict(os.environ, SBFS_LIB=CHECKED), capture_output=True, text=True, timeout=1800, cwd=ROOT)
    assert r.returncode == 0, r.stdout[-4000:] + r.stderr[-2000:]
    assert " passed" in r.stdout and "failed" not in r.stdout
