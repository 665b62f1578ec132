"""A block of the run kernel ends only when its asynchronous copies have arrived:
each return before the pieces that read the copied tables, the first drift's
among them, has a wait of its own before it.
"""
import os
import re

SRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "moldy_b200", "csrc", "run.cu")


def test_run_kernel_waits_for_its_copies_before_it_ends():
    src = open(SRC).read()
    i = re.search(r"^[^\n;/]*\bk_run\(", src, re.M).start()
    body = re.sub(r"//[^\n]*", "", src[i:src.index("\n}\n", i)])
    drift = body.index("if (h == 0) {")
    end = body.index("if (h == 2 * a.m + 1) {", drift)       # the next piece
    upto = body[:end]
    returns = [m.start() for m in re.finditer(r"\breturn;", upto)]
    assert len(returns) >= 2
    for r in returns:
        assert re.search(r"copies_arrived\(\);\s*$", upto[:r]), upto[max(0, r - 200):r + 8]
