"""BlockScheduler from C++ (tests/cpp/scheduler_test.cpp, built by the package's Makefile)."""
import os
import subprocess

import pytest

from _support import ROOT, load_package

pytestmark = pytest.mark.gpu
CSRC = os.path.join(ROOT, "gretacore-v3_b200", "csrc")


@pytest.mark.parametrize("check", ["norm_out", "copy_rows", "gave_up", "tensor_parallel"])
def test_scheduler(check):
    pkg = load_package()
    pkg.build()
    pkg.ffi.require_device()
    res = subprocess.run(["make", "-s", "-C", CSRC, "scheduler_test"], stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True)
    assert res.returncode == 0, res.stdout[-3000:]
    res = subprocess.run([os.path.join(CSRC, "..", "build", "scheduler_test"), check], stdout=subprocess.PIPE, stderr=subprocess.STDOUT, text=True, timeout=300)
    assert res.returncode == 0, res.stdout[-3000:]
