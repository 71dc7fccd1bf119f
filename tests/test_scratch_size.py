"""The size rules of the matcher's guessed buffers, run over an allocator with a
limit: a refused size is not tried again, a buffer that serves is kept."""
import os
import subprocess

from tests.conftest import ROOT


def test_rules_over_a_limited_allocator(tmp_path):
    exe = str(tmp_path / "check")
    subprocess.check_call([os.environ.get("CXX", "g++"), "-O1", "-std=c++17", "-Wall", "-o", exe,
                           os.path.join(ROOT, "tests", "scratch_size_check.cc")])
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
