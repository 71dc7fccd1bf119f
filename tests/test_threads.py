"""Host work on threads (bulk merge and sort at consolidation) when the system
refuses threads: the caller does what is left, nothing ends the process."""
import os
import subprocess

from tests.conftest import ROOT


def test_refused_threads(tmp_path):
    exe = str(tmp_path / "check")
    subprocess.check_call([os.environ.get("CXX", "g++"), "-O1", "-std=c++17", "-Wall", "-o", exe,
                           os.path.join(ROOT, "tests", "threads_check.cc"), "-lpthread"])
    r = subprocess.run([exe], capture_output=True, text=True)
    assert r.returncode == 0, (r.returncode, r.stdout, r.stderr)
