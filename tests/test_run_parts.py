"""The host threads of a stream build (RunParts): short of memory while they
are started, those there are do all the work; a part's exception is thrown
again when all have ended."""
import os
import subprocess

from conftest import TESTS, _cuda_include


def test_run_parts_short_of_memory(tmp_path):
    out = str(tmp_path / "run_parts")
    r = subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I" + _cuda_include(),
                        os.path.join(TESTS, "run_parts.cc"), "-o", out],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    r = subprocess.run([out], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout == "ok\n", (r.returncode, r.stderr)
