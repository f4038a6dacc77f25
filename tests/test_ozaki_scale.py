"""Outputs of the digit-sliced complex128 passes are scaled without branches
where the row's and the matrix's exponents allow it (ev_ozaki.cuh): the same
bits as the general form, on the device and on the host."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    nvcc = shutil.which("nvcc")
    assert nvcc, "nvcc is required"
    exe = tmp_path_factory.mktemp("oz") / "test_ozscale"
    r = subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-std=c++17", "-O2",
                        "-I", str(ROOT / "everett_gb300" / "csrc"),
                        str(ROOT / "tests" / "cpp" / "test_ozscale.cu"), "-o", str(exe)],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    return exe


def run(program, where):
    r = subprocess.run([str(program), where], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
    assert ", 0 differ on the device, 0 on the host" in r.stdout


def test_scaled_on_the_host(program):
    run(program, "host")


@pytest.mark.gpu
def test_plain_scaling_equals_scaled(gpu, program):
    run(program, "device")
