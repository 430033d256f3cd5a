"""Host-built tables of the atoms-on-lanes kernels, the Y rows and the derivatives
(mld_gb300/csrc/bso4_tables.cpp), checked by tests/lane_tables_check.cc with the host compiler (no GPU), and
the benchmark's work model, which counts what those tables make the kernels do: every product of an
operand pair once for all its output layers, every row entry once."""
import os
import re
import shutil
import subprocess

import pytest

from test_tables import ROOT, _cuda_include


@pytest.fixture(scope="module")
def checker(tmp_path_factory):
    cxx, inc = shutil.which("g++") or shutil.which("c++"), _cuda_include()
    if not cxx or not inc:
        pytest.skip("needs a host C++ compiler and the CUDA headers")
    exe = str(tmp_path_factory.mktemp("lanes") / "lane_tables_check")
    r = subprocess.run([cxx, "-std=c++17", "-O1", "-I", os.path.join(ROOT, "include"), "-I", inc,
                        os.path.join(ROOT, "tests", "lane_tables_check.cc"),
                        os.path.join(ROOT, "mld_gb300", "csrc", "bso4_tables.cpp"), "-o", exe], capture_output=True, text=True)
    assert r.returncode == 0, r.stderr[-3000:]
    return exe


@pytest.mark.parametrize("j_max", [0.0, 0.5, 1.0, 1.5, 2.0, 2.5, 3.0, 3.5, 4.0, 4.5, 5.0])
def test_tables_and_work_model(checker, j_max):
    import bench
    r = subprocess.run([checker, str(j_max)], capture_output=True, text=True)
    assert r.returncode == 0 and r.stdout.startswith("ok"), r.stdout + r.stderr
    want = {k: int(v) for k, v in re.findall(r"(\w+)=(\d+)", r.stdout)}
    got = bench.contraction_counts(int(2 * j_max))
    assert {k: got[k] for k in want} == want
