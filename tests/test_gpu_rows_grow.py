"""A box that has shrunk needs longer rows: they are allocated anew between two
calls, and the next step has to build them before it reads them."""
import numpy as np
import pytest

from moldy_b200 import MoldySystem
from moldy_b200 import workloads as wl

pytestmark = pytest.mark.gpu

ARGS = ("x0", "x1", "x2", "b0", "b1", "b2")


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("n,step", [(8, "md_steps"), (8, "velocityverlet"), (43, "md_steps")])
def test_steps_after_the_rows_grew(gpu_lib, n, step, prec):
    w = wl.make_workload(n, sigma=0.03, temperature=50.0, ivol=1, nbrupdate=50, nnbrs=250, seed=4)
    g = MoldySystem.from_workload(w, precision=prec)
    g.md_init()
    g.md_steps(3)
    st = g.get_state()
    st["b0"] = 0.78 * w.b0                      # twice the density: rows of 48 entries do not hold it
    fresh = MoldySystem.from_workload(w, precision=prec)
    for s in (g, fresh):
        s.set_state(*[st[k] for k in ARGS], tgid=st["tgid"])
    pe = []
    for s in (g, fresh):
        if step == "md_steps":
            pe.append([t["pe"] for t in s.md_steps(4)])
        else:
            pe.append([s.velocityverlet()["pe"] for _ in range(4)])
    assert g.list_stats()["pairs"] > 24 * w.nm  # the rows did grow
    tol = 1e-10 if prec == "fp64" else 1e-6
    assert np.max(np.abs(np.array(pe[0]) - np.array(pe[1]))) < tol * np.max(np.abs(pe[1]))
    g.close()
    fresh.close()
