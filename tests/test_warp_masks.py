"""Warp-wide exchanges name the lanes that take part: __activemask() is whatever
happens to run together at that instruction, so a group that reduces under one call
and elects its storing lane under another may lose its result.  Where a mask has to
be taken (lanes leaving a loop at different times) it is taken once and held."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parents[1] / "binarytpm_gb300" / "csrc"


def test_active_masks_are_held():
    sources = [p for p in sorted(CSRC.iterdir()) if p.suffix in (".cu", ".cuh", ".h")]
    assert sources
    for p in sources:
        text = re.sub(r"//[^\n]*", "", p.read_text())
        for line in text.splitlines():
            if "__activemask()" in line:
                assert re.fullmatch(r"\s*const unsigned \w+ = __activemask\(\);\s*", line), f"{p.name}: {line.strip()}"
