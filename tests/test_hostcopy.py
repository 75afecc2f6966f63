"""Staged host copies (csrc/pt_hostcopy.cuh) on the host, against a stand-in for the CUDA runtime (tests/cpp/fake_cuda).

Each check is a function of tests/cpp/hostcopy_check.cpp, run in a process of its own.
"""
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("hostcopy") / "hostcopy_check")
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", os.path.join(ROOT, "tests", "cpp", "fake_cuda"), "-I",
                    os.path.join(ROOT, "lsystemeditor_b200", "csrc"), os.path.join(ROOT, "tests", "cpp", "hostcopy_check.cpp"),
                    "-o", out], check=True)
    return out


@pytest.mark.parametrize("name", ["forked_child", "staging_rule", "shared", "threads", "errors_and_plain_copies"])
def test_hostcopy(program, name):
    r = subprocess.run([program, name], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, f"exit {r.returncode}: {r.stdout}{r.stderr}"
