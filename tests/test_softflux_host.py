"""The integer face flux of the exact FP64 heat kernels (csrc/softflux.cuh), built for the host by
nvcc from the same source, against the host's own FP64 operations: bit for bit."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
REPO = os.path.dirname(HERE)


def _nvcc():
    for c in (os.environ.get("NVCC"), "/usr/local/cuda/bin/nvcc", shutil.which("nvcc")):
        if c and os.path.exists(c):
            return c
    return None


def test_soft_flux_has_the_hardware_bits(tmp_path):
    nvcc = _nvcc()
    if nvcc is None:
        pytest.skip("needs nvcc")
    exe = str(tmp_path / "softflux_host")
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-O2", "-std=c++17", "-Xcompiler",
                    "-ffp-contract=off", "-I", os.path.join(REPO, "include"),
                    "-I", os.path.join(REPO, "spatialops-threadfix_gb300", "csrc"),
                    os.path.join(HERE, "cpp", "softflux_host.cu"), "-o", exe], check=True)
    for seed in (1, 2):
        out = subprocess.run([exe, "4000000", str(seed)], check=True, capture_output=True, text=True).stdout
        r = {ln.split()[0]: int(ln.split()[1]) for ln in out.splitlines()}
        assert r["bad"] == 0 and r["uncovered"] == 0, out
        assert r["covered"] > r["cases"] // 2, out
