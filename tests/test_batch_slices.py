"""The geometry slices of a batch stay apart, whichever renderer laid them out
and whichever lets passes outgrow them (tests/batch_slices.cc)."""
import os
import subprocess

from conftest import TESTS, _cuda_include


def test_slices_stay_apart(tmp_path):
    out = str(tmp_path / "batch_slices")
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I" + _cuda_include(),
                        os.path.join(TESTS, "batch_slices.cc"), "-o", out],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([out], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout == "ok\n", (r.returncode, r.stderr)
