"""Which form of the mixed pair passes runs, compiled from the rules the
launchers use: the force pass keeps its tables in shared memory only from the
size on where that form was measured the faster, whatever the variant."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.abspath(__file__)), "..", "moldy_b200", "csrc")
PROGRAM = r"""
#include <cstdio>
#include "rules.h"
int main() {
    const int sizes[] = {2000, 99999, 100000, 524288, 810448, 849999, 850000, 2000000, 90000000};
    const int all_nodes[] = {3104, 6000, 6001};
    for (int nm : sizes)
        for (int nodes : all_nodes)
            std::printf("%d %d %d %d\n", nm, nodes, moldy::screen_in_smem(nm, nodes, 48, 24) ? 1 : 0,
                        moldy::forces_in_smem(nm, nodes, 48, 24) ? 1 : 0);
}
"""


def test_forms_by_size(tmp_path):
    gxx = "/usr/bin/g++" if os.path.exists("/usr/bin/g++") else shutil.which("g++")
    if not gxx:
        pytest.skip("no host compiler")
    src, exe = tmp_path / "rules.cpp", str(tmp_path / "rules")
    src.write_text(PROGRAM)
    subprocess.run([gxx, "-std=c++17", "-I", CSRC, str(src), "-o", exe], check=True)
    out = subprocess.run([exe], capture_output=True, text=True, check=True).stdout
    for line in out.splitlines():
        nm, nodes, screen, forces = map(int, line.split())
        fits = nodes <= 6000 and nm * 64 < 2 ** 32
        assert screen == (fits and nm >= 100000), line
        assert forces == (fits and nm >= 850000), line
    # the launchers take their forms from these two and from nothing else
    pairs = open(os.path.join(CSRC, "pairs.cu")).read()
    assert "const bool st = mixed && forces_in_smem(p.nm, t.nr, p.mid_cap, p.pair_cap);" in pairs
    assert "variant >= 0 ||" not in pairs
