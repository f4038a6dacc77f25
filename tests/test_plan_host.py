"""The pass planner (plan_passes, everett_gb300/csrc/ev_tile.cuh) on the host:
its passes against the rule written out, and its time per gate on long
circuits against short ones."""
import shutil
import subprocess
from pathlib import Path

import pytest

ROOT = Path(__file__).resolve().parents[1]
LIBDIR = ROOT / "everett_gb300"


@pytest.fixture(scope="module")
def program(engine, tmp_path_factory):
    nvcc = shutil.which("nvcc")
    assert nvcc, "nvcc is required"
    exe = tmp_path_factory.mktemp("plan") / "test_plan"
    r = subprocess.run([nvcc, "-gencode", "arch=compute_103a,code=sm_103a", "-std=c++17", "-O2",
                        "--expt-relaxed-constexpr", "-I", str(LIBDIR / "csrc"),
                        str(ROOT / "tests" / "cpp" / "test_plan.cu"), "-o", str(exe),
                        "-L", str(LIBDIR), "-leverett_gb300", "-Xlinker", f"-rpath,{LIBDIR}"],
                       capture_output=True, text=True)
    assert r.returncode == 0, r.stdout + r.stderr
    return exe


def test_passes_follow_the_rule(program):
    r = subprocess.run([str(program), "same"], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0 and ", 0 differ" in r.stdout, r.stdout + r.stderr


def test_planning_is_linear_in_the_gates(program):
    """400 000 gates take at most four times as long per gate as 10 000 (the
    longer list leaves the caches; a walk over all that is pending in every
    pass would take forty times as long), with every qubit in use and with an
    idle one."""
    for attempt in range(3):  # a machine at work may spoil one
        r = subprocess.run([str(program), "time"], capture_output=True, text=True, timeout=300)
        assert r.returncode == 0, r.stdout + r.stderr
        rows = [line.split() for line in r.stdout.splitlines()]
        assert len(rows) == 12
        slow = [row for row in rows if float(row[4]) > 4 * float(row[3])]
        if not slow:
            return
    assert not slow


@pytest.mark.parametrize("sms", [76, 132, 148, 152, 160, 304])
def test_default_tiles_follow_the_sms(program, sms):
    """complex128 tiles of 2^11 or 2^12 by how evenly this GPU's SMs share
    them: never 2^12 where it leaves an SM without a tile, 2^11 exactly where
    the fullest SM's excess shrinks by more than a tenth.  On 152 SMs the
    sizes measured: 19 and 21 qubits."""
    r = subprocess.run([str(program), "tiles", str(sms)], capture_output=True, text=True, timeout=60)
    assert r.returncode == 0, r.stderr
    bits = {int(n): (int(a), int(b)) for n, a, b in (line.split() for line in r.stdout.splitlines())}

    def excess(tiles):
        return -(-tiles // sms) * sms / tiles

    for n in range(19, 35):
        tiles = 1 << (n - 12)
        small = tiles < sms or excess(tiles) > 1.1 * excess(2 * tiles)
        assert bits[n][0] == (11 if small else 12), n
    if sms == 152:
        want = [8] * 17 + [10, 11, 12, 11] + [12] * 13
        assert [bits[n][0] for n in range(1, 35)] == want
    assert [bits[n][1] for n in range(1, 35)] == [8] * 15 + [10] * 4 + [12] * 3 + [13] * 12
