"""Host-side helpers of the engine (csrc/rw_host.h), compiled on their own."""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    exe = str(tmp_path_factory.mktemp("host") / "host_test")
    subprocess.run(["g++", "-std=c++17", "-O2", "-pthread", "-I", os.path.join(ROOT, "retainwall_code_b200", "csrc"),
                    os.path.join(ROOT, "tests", "cpp", "host_test.cpp"), "-o", exe], check=True)
    return exe


@pytest.mark.parametrize("check", ["contents", "no_memory", "export_pieces"])
def test_host_helper(program, check):
    r = subprocess.run([program, check], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, (r.returncode, r.stdout, r.stderr)
