"""Kernels that let the next pass start early hold their tensor memory first.

A pass's CTA may take its columns and then wait, without bound, for the pass
before it.  That pass must not itself be waiting for columns, so the
instruction that lets the next pass start comes after the allocation, in the
warp that allocates.  Read from the source: the order can't be seen from
outside, and a kernel that has it wrong may hang."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "everett_gb300" / "csrc"
ALLOC, NEXT = "tcgen05.alloc.", "griddepcontrol.launch_dependents"


def bodies(src):
    """Every function of a source file, comments taken out: name -> body."""
    src = re.sub(r"//[^\n]*", "", src)
    out = {}
    for m in re.finditer(r"\n(?:__device__|__global__)[^;{]*?\b(\w+)\(", src):
        depth, i = 0, src.index("{", m.end())
        start = i
        while True:
            depth += {"{": 1, "}": -1}.get(src[i], 0)
            i += 1
            if depth == 0:
                break
        out[m.group(1) + str(m.start())] = src[start:i]
    return out


def test_columns_are_held_before_the_next_pass_may_start():
    allocs = 0
    for path in sorted(CSRC.glob("*.cu*")):
        text = path.read_text()
        # the kernels reach both instructions through one helper
        helpers = {re.sub(r"\d+$", "", n): b for n, b in bodies(text).items()
                   if ALLOC in b and "__syncthreads" not in b}
        for name, body in bodies(text).items():
            for h, b in helpers.items():
                body = re.sub(r"\b%s\b(<[^;]*?>)?\(" % h, b + "(", body)
            if ALLOC not in body:
                continue
            allocs += 1
            if NEXT in body:
                assert body.index(ALLOC) < body.index(NEXT), (path.name, name)
    assert allocs >= 3
