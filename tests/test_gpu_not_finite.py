"""Positions that are not finite (a run that blew up) have no link cell: the
call ends with an error, and the engine goes on with the next good state."""
import numpy as np
import pytest

from moldy_b200 import MoldySystem
from moldy_b200 import workloads as wl
from moldy_b200._lib import MoldyError

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("value,atoms", [(np.nan, [17]), (np.inf, [0, 1457]), (-np.inf, [5]), (np.nan, slice(None))])
def test_position_without_a_cell(gpu_lib, prec, value, atoms):
    w = wl.make_workload(9, sigma=0.05, temperature=300.0, ivol=1, nbrupdate=3, seed=3)
    g = MoldySystem.from_workload(w, precision=prec)
    pe, f = g.force()["pe"], g.forces()
    x = w.x0.copy()
    x[atoms, 1] = value
    for call in (g.linkup, g.relink):
        g.set_state(x0=x)
        call()
        with pytest.raises(MoldyError, match="not a finite"):
            g.force()
        g.set_state(x0=w.x0)
        out = g.force()
        assert abs(out["pe"] - pe) < 1e-9 * abs(pe) and np.max(np.abs(g.forces() - f)) < 1e-6 * np.max(np.abs(f))
    g.close()


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_run_that_blows_up(gpu_lib, prec):
    w = wl.make_workload(9, sigma=0.05, temperature=300.0, ivol=1, nbrupdate=3, seed=3)
    w.x1 = w.x1.copy()
    w.x1[40] = np.nan
    g = MoldySystem.from_workload(w, precision=prec)
    g.md_init()
    with pytest.raises(MoldyError, match="not a finite"):
        g.md_steps(10)
    g.close()


@pytest.mark.parametrize("mode", ["list", "all"])
def test_pairs_without_a_distance_fall_in_no_bin(gpu_lib, mode):
    from moldy_b200 import analysis
    w = wl.make_workload(6, sigma=0.05, temperature=300.0, ivol=1, seed=3)
    g = MoldySystem.from_workload(w, precision="fp64")
    g.force()
    x = w.x0.copy()
    x[[3, 200], 0] = np.nan
    g.set_state(x0=x)
    got = analysis.rdf(g, 200, 50, mode)
    z = w.atomic_number.copy()
    z[[3, 200]] = 0                       # as if the two atoms were vacancies
    g.set_state(x0=w.x0, atomic_number=z)
    want = analysis.rdf(g, 200, 50, mode)
    assert np.array_equal(got["hist"], want["hist"]) and got["nclose"] == want["nclose"]
    g.close()
