"""Copies of a plan run on the plan's own stream.

That stream is a non-blocking one: the blocking copies of the runtime go through the legacy stream, which it is
not ordered with.  An array cleared on the plan's stream and filled by such a copy could end up cleared, and
a kernel launched after such a copy from pageable memory could start before the last of it had arrived."""
import re
from pathlib import Path

CSRC = Path(__file__).resolve().parent.parent / "visual_cortex_gb300" / "csrc"


def test_no_copies_on_the_legacy_stream():
    text = (CSRC / "pv1_plan.cu").read_text()
    code = re.sub(r"//[^\n]*", "", text)
    found = [m.group(0) for m in re.finditer(r"\bcudaMem(?:cpy|set)(?:2D|3D|ToSymbol|FromSymbol)?\s*\([^;]*;", code)]
    assert not found, found
