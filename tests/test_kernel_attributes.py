"""Kernel attributes are set on every device of a process, by one thread: the helper that
does so (the shipped header compiled for the host), and that the engine keeps no flag of its
own for the whole process."""
import os
import re
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(HERE, "..", "sphadjoint_gb300", "csrc")


def test_once_per_device(tmp_path):
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("g++ not found")
    exe = str(tmp_path / "once_check")
    subprocess.run([cxx, "-O2", "-std=c++17", "-pthread", "-I", CSRC,
                    os.path.join(HERE, "once_check.cpp"), "-o", exe], check=True)
    out = subprocess.run([exe], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0, out.stdout + out.stderr


def test_no_process_wide_flag_beside_kernel_attributes():
    for name in os.listdir(CSRC):
        with open(os.path.join(CSRC, name)) as f:
            text = f.read()
        if "cudaFuncSetAttribute" in text:
            assert not re.search(r"\bstatic bool \w+ *[=;]", text), name
            assert "OncePerDevice" in text, name
