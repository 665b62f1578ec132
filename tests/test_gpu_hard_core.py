"""Tables with an infinite hard core: no pair comes inside it, so it may not
reach any force, energy or density.  The passes evaluate whole batches of row
entries, and what pads a row's last batch has to add nothing whatever the table
holds.  Same results, bit for bit, as with a finite core.
"""
import numpy as np
import pytest

from moldy_b200 import MoldySystem
from moldy_b200 import workloads as wl

pytestmark = pytest.mark.gpu
CORE, NLOOKUP = 1.5, 4000


def _tables(core_v, core_d):
    r = np.linspace(0.0, 4.0, NLOOKUP + 1)
    rho = np.linspace(0.0, 1000.0, NLOOKUP + 1)
    d = np.clip(3.6 - r, 0.0, None)
    t = dict(vee=d ** 3, dvee=-3.0 * d ** 2, phi=d ** 2, dphi=-2.0 * d, emb=-np.sqrt(rho + 1.0),
             demb=-0.5 / np.sqrt(rho + 1.0))
    t["vee"][r < CORE], t["dvee"][r < CORE] = core_v, core_d
    return t


def _evaluate(w, prec, tables):
    g = MoldySystem.from_workload(w, precision=prec)
    g.set_tables(tables, rmin=0.0, rmax=4.0, rhomin=0.0, rhomax=1000.0)
    out = g.force()
    f, rho = g.forces(), g.density()["rho"]
    g.md_init()
    th = g.md_steps(6)
    x = g.get_state()["x0"]
    g.close()
    return out["pe"], out["tp"], f, rho, x, np.array([[t["pe"], t["ke"]] for t in th])


# runs and launches; 76^3 cells: the mixed passes with their tables in shared memory
@pytest.mark.parametrize("prec,n", [("fp64", 7), ("mixed", 7), ("fp64", 37), ("mixed", 42), ("mixed", 76)])
def test_hard_core_reaches_nothing(gpu_lib, prec, n):
    w = wl.make_workload(n, sigma=0.05, temperature=300.0, ivol=1, nbrupdate=4, seed=n)
    a = _evaluate(w, prec, _tables(np.inf, -np.inf))
    b = _evaluate(w, prec, _tables(50.0, -100.0))
    assert np.isfinite(a[2]).all() and np.isfinite(a[0])
    for p, q in zip(a, b):
        assert np.array_equal(p, q)


def test_every_variant_of_the_large_passes_gives_the_same_forces(gpu_lib):
    """877,952 atoms: both mixed passes with their tables in shared memory."""
    w = wl.make_workload(76, sigma=0.08, temperature=300.0, ivol=0, seed=5)
    g = MoldySystem.from_workload(w, precision="mixed")
    g.force()
    f, rho = g.forces(), g.density()["rho"]
    for v in range(8):
        g.set_variants(v, 0, v)
        g.force()
        assert np.array_equal(g.forces(), f) and np.array_equal(g.density()["rho"], rho), v
    g.close()
    g = MoldySystem.from_workload(w, precision="fp64")
    g.force()
    assert np.sqrt(np.mean(((g.forces() - f) @ w.b0.T) ** 2)) < 1e-5
    g.close()
