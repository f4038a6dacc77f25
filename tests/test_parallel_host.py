"""Host work of a batch (planning its circuits) starts no more threads than
it has circuits: thread starts dominated small batches of the request loop."""
import shutil
import subprocess
from pathlib import Path

ROOT = Path(__file__).resolve().parents[1]
CSRC = ROOT / "everett_gb300" / "csrc"


def test_threads_and_indices(tmp_path):
    gxx = shutil.which("g++")
    assert gxx, "g++ is required"
    exe = tmp_path / "test_parallel"
    subprocess.run([gxx, "-std=c++17", "-O2", "-Wall", "-Wextra", "-Werror", "-pthread", "-I", str(CSRC),
                    str(ROOT / "tests" / "cpp" / "test_parallel.cpp"), "-o", str(exe)],
                   check=True, capture_output=True, text=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stdout


def test_batches_plan_through_it():
    """No other place of the batched runner starts threads."""
    src = (CSRC / "ev_batch.cu").read_text()
    assert src.count("parallel_for(") == 1
    assert "std::vector<std::thread>" not in src and "std::thread(" not in src
