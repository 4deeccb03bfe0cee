"""The host logic behind batches and the mirror-group kernel on the CPU:
occastft_gb300/csrc/ocs_api.cpp compiled unchanged against the CUDA stand-in and
stand-in kernels that launch a batch class by class (tests/fake_cuda/)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
FAKE = os.path.join(ROOT, "tests", "fake_cuda")
CSRC = os.path.join(ROOT, "occastft_gb300", "csrc")
SOURCES = [os.path.join(CSRC, "ocs_api.cpp"), os.path.join(CSRC, "ocs_host.cpp"),
           os.path.join(FAKE, "fake_runtime.cpp"), os.path.join(FAKE, "batch_class_kernels.cpp"),
           os.path.join(FAKE, "batch_class_checks.cpp")]
CHECKS = ["classes", "one_request", "failed_launch", "tune_key"]


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    cxx = os.environ.get("CXX", "g++")
    if not shutil.which(cxx):
        pytest.skip("no C++ compiler")
    out = str(tmp_path_factory.mktemp("batch_classes") / "batch_classes")
    r = subprocess.run([cxx, "-std=c++17", "-O1", "-g", "-pthread", "-I" + FAKE, "-I" + CSRC,
                        "-I" + os.path.join(ROOT, "include")] + SOURCES + ["-o", out],
                       capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stderr[-4000:]
    return out


@pytest.mark.parametrize("check", CHECKS)
def test_batch_classes(exe, check):
    env = {k: v for k, v in os.environ.items() if not k.startswith("OCS_")}
    p = subprocess.run([exe, check], capture_output=True, text=True, timeout=300, env=env)
    assert p.returncode == 0 and f"ok {check}" in p.stdout, (p.stdout + p.stderr)[-3000:]
