"""The float quantisers of the encoders' kernels against the integer rules, on
the CPU (tests/quant_check.cu)."""
import os
import subprocess

from tests.test_packed_lanes import HERE, ROOT, nvcc


def test_every_step_and_coefficient(tmp_path):
    exe = str(tmp_path / "quant_check")
    subprocess.run([nvcc(), "-std=c++17", "-O2", "--expt-relaxed-constexpr", "-Wno-deprecated-gpu-targets", "-gencode",
                    "arch=compute_100a,code=sm_100a", "-o", exe, os.path.join(HERE, "quant_check.cu"),
                    os.path.join(ROOT, "oracle", "tcoracle.c")], check=True, timeout=300)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
    assert "mismatches 0" in r.stdout
