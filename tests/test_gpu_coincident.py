"""Two atoms at one point, in every FP64 pass: the density is that of the
table's first node, the energy is infinite (V(0) is), the two atoms' forces have
no direction, and the others' are theirs.  As the oracle has it."""
import numpy as np
import pytest

from moldy_b200 import MoldyBatch, MoldySystem
from moldy_b200 import workloads as wl
from tests.helpers import rel_norm_err

pytestmark = pytest.mark.gpu


def _workload(apart=0.0):
    w = wl.make_workload(5, sigma=0.05, temperature=0.0, ivol=1, seed=3)
    w.x0 = w.x0.copy()
    w.x0[17] = w.x0[16] + np.linalg.solve(w.b0, [apart, 0.0, 0.0])
    return w


def _check(w, o, pe, f, rho):
    assert pe == np.inf and o.force_out()["pe"] == np.inf
    want = o.forces()
    pair = ~np.isfinite(want).all(axis=1)
    assert np.array_equal(np.flatnonzero(pair), [16, 17])
    assert not np.isfinite(f[pair]).any()
    assert rel_norm_err(f[~pair], want[~pair]) < 1e-10
    assert rel_norm_err(rho, o.density()["rho"]) < 1e-10


# at one point, and inside the first interval of the tables (7e-4 A wide), whose lower node is infinite
@pytest.mark.parametrize("apart", [0.0, 3e-4])
def test_coincident_atoms(oracle_mod, gpu_lib, apart):
    w = _workload(apart)
    o = oracle_mod.from_workload(w, uselookup=True, threads=2)
    o.force()
    g = MoldySystem.from_workload(w, precision="fp64")
    _check(w, o, g.force()["pe"], g.forces(), g.density()["rho"])
    g.close()
    b = MoldyBatch.from_workloads([w, wl.make_workload(4, sigma=0.05, temperature=0.0, ivol=1, seed=4)])
    out = b.force()
    _check(w, o, out["pe"][0], b.split(b.forces())[0], b.split(b.density()["rho"])[0])
    assert np.isfinite(out["pe"][1]) and np.isfinite(b.split(b.forces())[1]).all()
    b.close()
