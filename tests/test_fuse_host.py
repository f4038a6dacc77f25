"""The fused planner multiplies its gates into a block's unitary with stated
roundings (everett_gb300/csrc/ev_fuse.h), the same on every host and with
every compiler: compiled as the engine is, without contraction, and with the
compiler's own."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
LIBDIR = ROOT / "everett_gb300"


@pytest.mark.parametrize("flags", ["-O2", "-O3,-ffp-contract=off", "-O3,-ffp-contract=fast", "-O0"])
def test_block_arithmetic_rounds_as_stated(engine, tmp_path, flags):
    nvcc = shutil.which("nvcc")
    assert nvcc, "nvcc is required"
    exe = tmp_path / "test_fuse"
    r = subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-std=c++17",
                        "-Xcompiler", flags, "-I", str(LIBDIR / "csrc"),
                        str(ROOT / "tests" / "cpp" / "test_fuse.cu"), "-o", str(exe),
                        "-L", str(LIBDIR), "-leverett_gb300", "-Xlinker", f"-rpath,{LIBDIR}"],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0 and ", 0 differ" in r.stdout, r.stdout + r.stderr
