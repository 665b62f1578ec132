"""Read-only loads (ld.global.nc: ldg4, ldg8f, __ldg) and __restrict__ const
pointers are undefined for memory that the same launch writes.  The tile
screen runs inside the launch that writes the slots' positions, so its
functions load them plainly.
"""
import os
import re

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "moldy_b200", "csrc")


def _function(src, name):
    """Signature and body of the function definition `name`."""
    m = re.search(r"^[^\n;/]*\b%s\(" % name, src, re.M)
    assert m, name
    i = src.index("{", m.end())
    depth, k = 1, i + 1
    while depth:
        depth += {"{": 1, "}": -1}.get(src[k], 0)
        k += 1
    return src[m.start():k]


def test_tile_screen_loads_what_its_launch_wrote():
    src = open(os.path.join(CSRC, "batch.cu")).read()
    for name in ("slot_record", "stage_tile", "candidate", "inside_list", "screen_cell", "prepare_system"):
        f = _function(src, name)
        assert not re.search(r"\b(ldg4|ldg8f|__ldg)\(", f), name
        assert not re.search(r"const double4 \*__restrict__", f), name
    assert ".nc" not in _function(src, "load_slot")
