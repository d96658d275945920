"""A refused launch (bulk_b200/csrc/bk_common.cuh, launch_overlapped) is reported
by its own call alone.  Runs on the host, against a stand-in for the runtime's
launch and its last error."""
from __future__ import annotations

import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
NVCC = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"


@pytest.mark.skipif(not Path(NVCC).exists(), reason="needs nvcc")
def test_failed_launch_leaves_no_error_behind(tmp_path):
    exe = tmp_path / "launch_error_check"
    subprocess.run([NVCC, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "--expt-relaxed-constexpr",
                    "-Xlinker", "--wrap=cudaLaunchKernelExC", "-Xlinker", "--wrap=cudaGetLastError",
                    f"-I{ROOT / 'include'}", f"-I{ROOT / 'bulk_b200' / 'csrc'}",
                    str(ROOT / "tests" / "host" / "launch_error_check.cu"), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and r.stdout.strip() == "ok", r.stdout + r.stderr
