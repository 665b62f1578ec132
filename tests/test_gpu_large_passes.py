"""The pair passes of large systems: the mixed ones with their tables in shared
memory (from 100,000 atoms on), and the FP64 ones, against the oracle at a
size that fills no block evenly, in every compiled variant, and with tables
that do not fit in shared memory or do not end in zeros.

Tolerances: FP64 terms differ from the oracle's by a few ulp each (root and
inverse from one reciprocal square root), 1e-10 norm-wise as for every FP64
force call; mixed is held to its gate, 1e-5 eV/A RMS and 1e-6 eV per atom.
"""
import numpy as np
import pytest

from moldy_b200 import workloads as wl
from tests.helpers import rel_norm_err

pytestmark = pytest.mark.gpu

N = 37          # 101,306 atoms: 131.9 blocks of 768, 98.9 of 1024


@pytest.fixture(scope="module")
def reference(oracle_mod):
    strain = [[0.004, 0.01, -0.006], [0.01, -0.003, 0.008], [-0.006, 0.008, 0.002]]
    w = wl.make_workload(N, sigma=0.12, temperature=900.0, ivol=0, seed=41, strain=strain)
    w.atomic_mass = w.atomic_mass.copy()
    w.atomic_mass[[5, 77777]] = 0.04            # a pair of them has no virial
    o = oracle_mod.from_workload(w, uselookup=True, threads=16)
    o.force()
    return w, o.force_out(), o.forces(), o.density()


def _check(g, ref, prec):
    w, fo, f, rho = ref
    out = g.force()
    if prec == "fp64":
        assert rel_norm_err(g.forces(), f) < 1e-10
        assert rel_norm_err(out["tp"], fo["tp"]) < 1e-10 and abs(out["pe"] - fo["pe"]) < 1e-10 * abs(fo["pe"])
        assert rel_norm_err(g.density()["rho"], rho["rho"]) < 1e-10
    else:
        d = (g.forces() - f) @ w.b0.T
        assert np.sqrt(np.mean(d ** 2)) < 1e-5 and abs(out["pe"] - fo["pe"]) < 1e-6 * w.nm
        assert rel_norm_err(out["tp"], fo["tp"]) < 1e-4


@pytest.mark.parametrize("prec", ["mixed", "fp64"])
def test_every_variant_follows_the_oracle(gpu_lib, reference, prec):
    from moldy_b200 import MoldySystem
    g = MoldySystem.from_workload(reference[0], precision=prec)
    _check(g, reference, prec)                  # the variants chosen by size
    for v in range(8):
        g.set_variants(v, 0, v)
        _check(g, reference, prec)
    g.close()


@pytest.mark.parametrize("nlookup,tail", [(20000, 0.0), (4000, 0.02)])
def test_tables_past_the_shared_memory_and_with_a_tail(oracle_mod, gpu_lib, nlookup, tail):
    """20,000 intervals (more nodes than the passes stage) and a table cut at
    3.2 A whose last node is not zero."""
    from moldy_b200 import MoldySystem
    w = wl.make_workload(N, sigma=0.05, temperature=0.0, ivol=1, seed=3)
    r = np.linspace(1.2, 3.2, nlookup + 1)
    rho = np.linspace(0.0, 10000.0, nlookup + 1)
    t = dict(vee=(3.2 - r) ** 3 + tail, dvee=-3.0 * (3.2 - r) ** 2 - tail, phi=(3.2 - r) ** 2 + tail,
             dphi=-2.0 * (3.2 - r) - tail, emb=-np.sqrt(rho + 1.0), demb=-0.5 / np.sqrt(rho + 1.0))
    rng = dict(rmin=1.2, rmax=3.2, rhomin=0.0, rhomax=10000.0)
    o = oracle_mod.from_workload(w, uselookup=True, threads=16)
    o.set_tables(t, **rng)
    o.force()
    fo, f = o.force_out(), o.forces()
    for prec in ("mixed", "fp64"):
        g = MoldySystem.from_workload(w, precision=prec)
        g.set_tables(t, **rng)
        out = g.force()
        if prec == "fp64":
            assert rel_norm_err(g.forces(), f) < 1e-10 and abs(out["pe"] - fo["pe"]) < 1e-10 * abs(fo["pe"])
        else:
            assert np.sqrt(np.mean(((g.forces() - f) @ w.b0.T) ** 2)) < 1e-5
            assert abs(out["pe"] - fo["pe"]) < 1e-6 * w.nm
        g.close()
