"""A program that calls cudaDeviceReset between uses of the library (tests/reset_driver.cu):
the device pool of the ended context is not used again."""
import os
import subprocess

import pytest

from conftest import ROOT

pytestmark = pytest.mark.gpu

NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")


def test_use_after_a_device_reset(hmg, cuda, tmp_path):
    exe, libdir = str(tmp_path / "reset_driver"), os.path.join(ROOT, "hmglib_b200")
    subprocess.run([NVCC, "-gencode", "arch=compute_100a,code=sm_100a", "-I", os.path.join(ROOT, "include"),
                    os.path.join(ROOT, "tests", "reset_driver.cu"), "-o", exe, "-L", libdir, "-lhmg",
                    "-Xlinker", f"-rpath,{libdir}"], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and "equal" in r.stdout, (r.returncode, r.stdout + r.stderr)
