"""The v2 decoder's host side on the CPU (tests/decoder_host_check.cpp): the
sizes, pointers and vectors it hands to the kernel, for streams whose pictures
change size and decoders created for another size than the stream's."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")


@pytest.fixture(scope="module")
def exe(tmp_path_factory):
    if not os.path.exists(os.path.join(CUDA, "include", "cuda_runtime.h")):
        pytest.skip("CUDA headers not found")
    out = str(tmp_path_factory.mktemp("decoder") / "decoder_host_check")
    subprocess.run(["g++", "-O1", "-std=c++17", "-w", "-I", os.path.join(CUDA, "include"), "-o", out,
                    os.path.join(HERE, "decoder_host_check.cpp"),
                    os.path.join(ROOT, "tcodec_b200", "csrc", "tcb_entropy.cpp"), "-lpthread"], check=True, timeout=300)
    return out


def run(exe, *args):
    r = subprocess.run([exe] + [str(a) for a in args], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout + r.stderr


@pytest.mark.parametrize("form", ["sizes", "reorder"])
@pytest.mark.parametrize("created", [(0, 0), (96, 80), (8, 8), (95, 79), (640, 360)])
@pytest.mark.parametrize("sizes", [(96, 80), (96, 80, 96, 16), (96, 16, 96, 80), (64, 64, 200, 136, 72, 8), (8, 8, 130, 70)])
def test_the_kernel_gets_the_frames_size(exe, form, created, sizes):
    run(exe, form, *created, *sizes)


@pytest.mark.parametrize("form", ["status", "status_key"])
@pytest.mark.parametrize("lost", [0, 1, 2, 4, 5, 7])      # before, at and after the fourth reference
def test_a_packet_that_fails_in_the_kernel_leaves_no_trace(exe, form, lost):
    run(exe, form, 0, 0, 72, 40, 9, lost)
