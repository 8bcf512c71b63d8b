"""The counters that the block-decided sweep's warps share
(csrc/block_turns.h), checked in a host program."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_block_turns(tmp_path):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("no host compiler")
    exe = str(tmp_path / "block_turns")
    subprocess.run([cxx, "-std=c++17", "-O2", os.path.join(ROOT, "tests", "integration", "block_turns.cc"), "-o", exe],
                   check=True)
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
