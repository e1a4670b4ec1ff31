"""The status that a call returns for the flags its kernels set (csrc/common.cuh), on the host: a
wait that ran out is NRG_ERR_TIMEOUT (9) whatever else is set, a secular root or a value that is
not finite NRG_ERR_NUMERIC (8), a bad index NRG_ERR_INVALID (1)."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
NVCC = os.environ.get("NVCC", "/usr/local/cuda/bin/nvcc")


@pytest.mark.skipif(not os.path.exists(NVCC) and shutil.which("nvcc") is None, reason="nvcc not available")
def test_status_of_device_flags(tmp_path):
    src, exe = tmp_path / "status.cu", str(tmp_path / "status")
    src.write_text('#include "common.cuh"\n'
                   "int main() { for (int f = 0; f < 32; ++f) std::printf(\"%d \", device_status_code(f)); }\n")
    subprocess.run([NVCC if os.path.exists(NVCC) else "nvcc", "-std=c++17", "-Wno-deprecated-gpu-targets", "-o", exe,
                    str(src), "-I", os.path.join(ROOT, "nrg-mpi_b200", "csrc")], check=True, capture_output=True, timeout=600)
    got = [int(x) for x in subprocess.run([exe], capture_output=True, text=True, check=True).stdout.split()]
    assert got == [0 if f == 0 else 9 if f & 16 else 8 if f & 12 else 1 for f in range(32)]
