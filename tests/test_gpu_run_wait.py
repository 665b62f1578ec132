"""A grid barrier of a run that the other blocks do not reach in time ends the
call with an error, and the engine runs on from the next state.  The limit is
lowered until no wait fits in it: every block but the last to arrive gives up
at its first poll, and the kernel ends by itself."""
import numpy as np
import pytest

from moldy_b200 import MoldySystem
from moldy_b200 import workloads as wl
from moldy_b200._lib import MoldyError

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("n,ivol", [(10, 1), (17, 0)])
def test_barrier_that_gives_up(gpu_lib, n, ivol, prec):
    w = wl.make_workload(n, sigma=0.08, temperature=900.0, ivol=ivol, press_gpa=1.0, nbrupdate=50, seed=2)
    g = MoldySystem.from_workload(w, precision=prec)
    g.md_init()
    want = g.md_steps(30)
    x = g.get_state()["x0"]
    g.close()
    g = MoldySystem.from_workload(w, precision=prec)
    g.md_init()
    g.set_run_wait(0, 0.0)
    with pytest.raises(MoldyError, match="gave up waiting"):
        g.md_steps(30)
    g.set_run_wait()
    g.set_state(w.x0, w.x1, w.x2, w.b0, w.b1, w.b2, w.atomic_number, w.atomic_mass, w.del2, w.tgid)
    g.set_ntc(0)
    g.md_init()
    got = g.md_steps(30)
    pe = np.array([[t["pe"], t["ke"]] for t in want])
    tol = 1e-11 if prec == "fp64" else 1e-7
    assert np.max(np.abs(np.array([[t["pe"], t["ke"]] for t in got]) - pe)) < tol * np.max(np.abs(pe))
    assert np.max(np.abs(g.get_state()["x0"] - x)) < tol
    g.close()


def test_limits_are_checked(gpu_lib):
    g = MoldySystem.from_workload(wl.make_workload(5))
    for polls, seconds in ((-1, 1.0), (1 << 40, 1.0), (10, -1.0), (10, 1e9), (10, float("nan"))):
        with pytest.raises(MoldyError, match="out of range"):
            g.set_run_wait(polls, seconds)
    g.close()
