"""Out of host memory while streams are parsed and their draws added, in the
caller's thread or in one of the others: a status, no exception and no abort
(tests/build_memory.cc)."""
import os
import subprocess

import pytest

from conftest import TESTS, _cuda_include
from skity_gb300 import scene as S
from test_build_streams import _one_large


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("build_memory") / "build_memory")
    r = subprocess.run(["g++", "-std=c++17", "-O2", "-pthread", "-I" + _cuda_include(),
                        os.path.join(TESTS, "build_memory.cc"), "-o", out],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return out


@pytest.mark.parametrize("kind,threads,step", [("many", 1, 29), ("many", 4, 37), ("large", 3, 41)])
def test_short_of_memory_is_a_status(program, tmp_path, kind, threads, step):
    bufs = ([_one_large(1400)] if kind == "large" else
            [sc.to_bytes() for sc in S.config3(n_canvases=16, scale=0.05)])
    files = []
    for i, b in enumerate(bufs):
        files.append(str(tmp_path / f"{i}.bin"))
        with open(files[-1], "wb") as f:
            f.write(b)
    r = subprocess.run([program, str(threads), str(step), *files], capture_output=True, text=True,
                       timeout=300)
    assert r.returncode == 0, (r.returncode, r.stderr)
    whole, cut = (int(v) for v in r.stdout.split())
    assert cut > 0.8 * (whole // step), (whole, cut)
