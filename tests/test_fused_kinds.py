"""The op-by-op fused pass on the host (CPU only), through
tests/fused_kinds_check.cu: it takes every kind of operation that its kernel
applies and reports the dense gates, which it would otherwise leave out."""
import os
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_unknown_kinds_are_refused(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not available")
    exe = str(tmp_path / "fused_kinds_check")
    subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=compute_100a", "-std=c++17", "--expt-relaxed-constexpr",
                    "-I", os.path.join(ROOT, "include"), "-I", os.path.join(ROOT, "tmfqsfullstate_b200", "csrc"),
                    "-o", exe, os.path.join(ROOT, "tests", "fused_kinds_check.cu")], check=True, timeout=600)
    out = subprocess.run([exe], capture_output=True, text=True, check=True, timeout=60).stdout.split("\n")[:-1]
    got = {int(f[1]): f[4] for f in map(str.split, out)}
    assert len(out) == 20
    assert got == {k: "refused" if k >= 8 else "accepted" for k in range(10)}
    assert all(line.split()[4] == got[int(line.split()[1])] for line in out)
