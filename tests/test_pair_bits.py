"""The FP64 <-> FP32-pair conversions on bit patterns against the conversions themselves: the same bits for
random patterns of the whole range, ties of the high and of the low part, values below the normal floats,
around the largest one, infinities, NaN and zeros of both signs."""
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "adaptive-multiresolution-dg_gb300", "csrc")


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    exe = str(tmp_path_factory.mktemp("pair_bits") / "pair_bits_check")
    subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-std=c++17", "-O3", "-I", CSRC, "-o", exe,
                    os.path.join(HERE, "pair_bits_check.cu")], check=True)
    return exe


def run(program, where, n):
    out = subprocess.run([program, where, str(n)], capture_output=True, text=True, timeout=300)
    assert out.returncode == 0, out.stdout + out.stderr
    assert out.stdout.split()[2] == "0"


def test_conversions_on_the_host(program):
    run(program, "host", 4_000_000)


@pytest.mark.gpu
def test_conversions_on_the_device(program):
    run(program, "device", 40_000_000)
