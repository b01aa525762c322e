"""llg_integrator_init takes over the vectors of the integrator it replaces.
On the CPU, with a fake CUDA runtime that fails each fallible call in turn
(tests/native/integrator_init_check.cpp): a failed call leaves the old integrator
whole or the context without one, and leaks nothing."""
import os
import shutil
import subprocess

import pytest

from conftest import PKG, REPO

CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


@pytest.mark.skipif(shutil.which("g++") is None or not os.path.isdir(os.path.join(CUDA, "include")),
                    reason="g++ or the CUDA headers are missing")
def test_failed_calls(tmp_path):
    # the file with a host-only stand-in for the kernel launches' header
    shutil.copy(os.path.join(PKG, "csrc", "integrator.cu"), tmp_path)
    (tmp_path / "launch.h").write_text("struct PdlScope { explicit PdlScope(bool) {} };\ninline void pdl_break() {}\n")
    exe = tmp_path / "integrator_init_check"
    subprocess.run(["g++", "-std=c++17", "-O1", "-w", "-I" + str(tmp_path), "-I" + os.path.join(PKG, "csrc"),
                    "-I" + os.path.join(CUDA, "include"),
                    os.path.join(REPO, "tests", "native", "integrator_init_check.cpp"), "-o", str(exe),
                    "-Wl,--unresolved-symbols=ignore-all"], check=True, capture_output=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert out.returncode == 0, out.stdout + out.stderr
