"""Fused runs of velocity-Verlet steps (moldy_b200/csrc/run.cu) against the
oracle, at the sizes where the lanes per atom change (the last atom of one
shape, the first of the next), for a fixed, a fully flexible and a z-only box.

Tolerances, from the size of what differs: FP64 runs add the same terms in
another order, 1e-15 relative per sum, and 12 steps of 1 fs do not amplify it
beyond rounding of positions: thermo 1e-11 relative, positions 1e-11 A.  Mixed
runs carry the FP32 pair terms' 1e-5 eV/A force gate: 12 steps of 1 fs move an
atom by at most 12^2 * 1e-5 * dt^2 / 2m = 2e-7 A off, and the energy gate is
1e-6 eV per atom.
"""
import numpy as np
import pytest

from moldy_b200 import workloads as wl

pytestmark = pytest.mark.gpu


def _follow(oracle_mod, w, prec, steps, skins=None):
    from moldy_b200 import MoldySystem
    g = MoldySystem.from_workload(w, precision=prec)
    if skins:
        g.set_mid_skin(skins[0])
        g.set_outer_skin(skins[1])
    o = oracle_mod.from_workload(w, uselookup=True, threads=8)
    o.md_init()
    g.md_init()
    before = g.kernel_stats()["forces"][1]
    tg = g.md_steps(steps)
    fused = g.kernel_stats()["forces"][1] - before < steps
    to = [o.md_step() for _ in range(steps)]
    so, sg = o.get_state(), g.get_state()
    pe = np.array([[t[k] for k in ("pe", "ke", "te", "vol")] for t in tg])
    po = np.array([[t[k] for k in ("pe", "ke", "te", "vol")] for t in to])
    if prec == "fp64":
        assert np.max(np.abs(pe - po) / np.abs(po)) < 1e-11
        assert np.max(np.abs((sg["x0"] - so["x0"]) @ w.b0.T)) < 1e-11
        assert np.max(np.abs(sg["x1"] - so["x1"])) < 1e-12 * np.max(np.abs(so["x1"])) * steps
        assert np.max(np.abs(g.forces() - o.forces())) < 1e-10 * np.max(np.abs(o.forces()))
        assert np.max(np.abs(g.density()["rho"] - o.density()["rho"])) < 1e-10 * np.max(o.density()["rho"])
    else:
        assert np.max(np.abs(pe[:, :3] - po[:, :3])) < 1e-6 * w.nm
        assert np.max(np.abs((sg["x0"] - so["x0"]) @ w.b0.T)) < 2e-7
        f, fo = g.forces() @ w.b0.T, o.forces() @ w.b0.T
        assert np.sqrt(np.mean((f - fo) ** 2)) < 1e-5
    assert np.max(np.abs(sg["b0"] - so["b0"])) < (1e-11 if prec == "fp64" else 1e-7) * np.max(so["b0"])
    stats = g.list_stats()
    g.close()
    return fused, stats


# 16 lanes per atom up to 4,736 atoms, 8 up to 9,472, 4 up to 18,944, 2 up to
# 37,888, one beyond; from 75,777 on two rounds of atoms in mixed precision and
# launched passes in FP64
@pytest.mark.parametrize("n", [6, 13, 14, 16, 17, 21, 22, 26, 27, 34])
@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_run_follows_the_oracle_at_every_shape(oracle_mod, gpu_lib, n, prec):
    w = wl.make_workload(n, sigma=0.08, temperature=900.0, ivol=0, press_gpa=1.0, nbrupdate=5, seed=n)
    fused, _ = _follow(oracle_mod, w, prec, 12)
    assert fused == (prec == "mixed" or w.nm <= 75776)


@pytest.mark.parametrize("ivol", [1, 4])
@pytest.mark.parametrize("prec", ["fp64", "mixed"])
def test_run_boxes_light_atoms_and_list_builds(oracle_mod, gpu_lib, ivol, prec):
    """A fixed and a z-only box, thin skins (several builds of both lists
    inside the runs), and a few atoms below the mass limits."""
    w = wl.make_workload(7, sigma=0.08, temperature=1500.0, ivol=ivol, press_gpa=0.5, nbrupdate=50, seed=5 + ivol)
    w.atomic_mass = w.atomic_mass.copy()
    w.atomic_mass[[3, 200, 685]] = 0.04
    w.x1 = w.x1.copy()
    w.x1[[3, 200, 685]] = 0.0
    w.del2 = np.where(w.atomic_mass > 0.1, w.deltat ** 2 / (2.0 * w.atomic_mass), 0.0)
    fused, stats = _follow(oracle_mod, w, prec, 30, skins=(0.04, 0.44))
    assert fused and stats["mid_builds"] >= 4


def test_run_without_records_gives_the_same_state(gpu_lib):
    """md_steps with and without thermo records, bit for bit."""
    from moldy_b200 import MoldySystem
    w = wl.make_workload(9, sigma=0.08, temperature=900.0, ivol=0, nbrupdate=7, seed=2)
    out = []
    for thermo in (True, False):
        g = MoldySystem.from_workload(w, precision="mixed")
        g.md_init()
        g.md_steps(25, thermo=thermo)
        g.md_steps(2, thermo=thermo)
        out.append((g.get_state(), g.forces()))
        g.close()
    for k in ("x0", "x1", "x2", "b0", "b1"):
        assert np.array_equal(out[0][0][k], out[1][0][k]), k
    assert np.array_equal(out[0][1], out[1][1])
