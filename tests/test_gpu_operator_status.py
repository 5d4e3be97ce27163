"""Operator calls whose waits for bulk copies run out (the flag is raised by
the test, no copy is late): tests/compat/operator_status_driver.cu."""
import os
import shutil
import subprocess

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu


def test_late_copy_fails_its_own_call_only(cb, tmp_path):
    nvcc = shutil.which("nvcc")
    if nvcc is None:
        pytest.skip("no nvcc")
    exe = tmp_path / "operator_status_driver"
    libdir = os.path.join(ROOT, "cvc_b200")
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17",
                    "--expt-relaxed-constexpr", "-o", str(exe),
                    os.path.join(ROOT, "tests/compat/operator_status_driver.cu"),
                    "-I" + os.path.join(ROOT, "include"), "-L" + libdir, "-lcvcb200",
                    "-Xlinker", "-rpath," + libdir], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert out.returncode == 0, out.stderr
    assert out.stdout.split() == ["1", "1", "1"]
