"""Rules of the kernels' sources that no result shows."""
import glob
import os
import re

from synaptix_b200.csrc.build import CSRC_DIR

SOURCES = {os.path.basename(f): open(f).read() for f in sorted(glob.glob(os.path.join(CSRC_DIR, "*.cu*")))}


def body_around(text, at):
    """The function whose body holds ``text[at]``: the last one that begins at the start of a line before it."""
    begin = max(m.start() for m in re.finditer(r"(?m)^(template|__global__|__device__)", text[:at]))
    depth = 0
    for i in range(text.index("{", text.index(")", begin)), len(text)):
        depth += {"{": 1, "}": -1}.get(text[i], 0)
        if depth == 0:
            return text[begin:i + 1]


def test_loads_from_tensor_memory_end_their_helper():
    """The registers of ``tcgen05.ld`` hold their values after ``tcgen05.wait::ld``: a helper that loads reads none of them, and
    leaves even a conversion to its caller, behind the wait."""
    found = 0
    for name, text in SOURCES.items():
        for m in re.finditer(r'"tcgen05\.ld\.', text):
            body = body_around(text, m.start())
            rest = body[body.index("tcgen05.ld."):]
            assert re.fullmatch(r"\s*\}", rest[rest.index(");") + 2:]), (name, body[:80])
            found += 1
    assert found >= 3


def test_tensor_memory_is_taken_before_the_next_kernel_is_let_in():
    """A block that lets the next kernel in (any warp's trigger does) while it still waits for tensor memory could wait for a
    block that waits for it."""
    found = 0
    for name, text in SOURCES.items():
        for m in re.finditer(r'"tcgen05\.alloc\.', text):
            body = body_around(text, m.start())
            rest = body[body.index("tcgen05.alloc."):]
            between = rest[:rest.index("pdl_trigger()")]
            assert "__syncthreads()" in between or "cluster_sync_all()" in between, (name, body[:80])
            found += 1
    assert found >= 5
