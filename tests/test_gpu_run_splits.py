"""How the steps of a run are split into calls, and through which entry points
they go, changes no bit of the state, the forces or the thermo records: fixed,
fully flexible and z-only boxes, with and without the thermostat, at sizes with
16, 4, 1 and 1/2 lanes per atom, across half-list builds and relinks."""
import numpy as np
import pytest

from moldy_b200 import MoldySystem
from moldy_b200 import workloads as wl

pytestmark = pytest.mark.gpu

STATE = ("x0", "x1", "x2", "b0", "b1", "b2", "tgid")


def _engine(w, prec, nose):
    g = MoldySystem.from_workload(w, precision=prec)
    if nose:
        g.set_thermostat(nose, 0.5 * 3 * w.nm * 0.0776)
    g.md_init()
    return g


def _outcome(g, records):
    d = g.density()
    s = g.get_state()
    out = {k: np.asarray(s[k]) for k in STATE}
    out.update(f=g.forces(), rho=d["rho"], records=np.array([list(r.values()) for r in records]))
    g.close()
    return out


def _same(a, b, what):
    for k in a:
        assert np.array_equal(a[k], b[k]), (what, k, np.max(np.abs(a[k] - b[k])))


def _steps(w, prec, nose, split, profile=False):
    g = _engine(w, prec, nose)
    if profile:
        g.set_profiling(True)
    records = []
    for n in split:
        records += g.md_steps(n)
    return _outcome(g, records)


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("n,ivol,nose", [(6, 0, 0.0), (6, 1, 0.0), (6, 4, 0.0), (6, 1, 5.0), (6, 0, 5.0), (17, 0, 0.0),
                                         (27, 1, 0.0), (27, 0, 0.0), (36, 0, 0.0), (43, 0, 5.0)])
def test_split_changes_no_bit(gpu_lib, n, ivol, nose, prec):
    w = wl.make_workload(n, sigma=0.08, temperature=900.0, ivol=ivol, press_gpa=1.0, nbrupdate=5, seed=n + ivol)
    want = _steps(w, prec, nose, [13])
    for split in ([1] * 13, [2, 1, 4, 6], [5, 5, 3]):
        _same(want, _steps(w, prec, nose, split), split)
    _same(want, _steps(w, prec, nose, [6, 7], profile=True), "profiled")


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("fs", [0.5, 0.34, 0.8])
def test_split_under_the_thermostat_changes_no_bit(gpu_lib, fs, prec):
    """scalev every second or third step (runs between), and at most steps."""
    w = wl.make_workload(8, sigma=0.08, temperature=900.0, ivol=0, nbrupdate=7, seed=3, dt_fs=fs)
    want = _steps(w, prec, 5.0, [23])
    for split in ([1] * 23, [2, 1, 4, 6, 10]):
        _same(want, _steps(w, prec, 5.0, split), split)


@pytest.mark.parametrize("prec", ["fp64", "mixed"])
@pytest.mark.parametrize("n,ivol", [(6, 0), (6, 1), (43, 0)])
def test_velocity_verlet_takes_the_same_steps(gpu_lib, n, ivol, prec):
    """The reference's own loop: velocityverlet, update_therm_avs, relink; in
    runs and, at 159,014 atoms, in launches."""
    w = wl.make_workload(n, sigma=0.08, temperature=900.0, ivol=ivol, press_gpa=1.0, nbrupdate=5, seed=9)
    want = _steps(w, prec, 0.0, [13])
    g = _engine(w, prec, 0.0)
    for _ in range(13):
        out = g.velocityverlet()
        g.update_therm_avs()
        if out["ntc"] == 0:
            g.relink()
    got = _outcome(g, [])
    del want["records"], got["records"]
    _same(want, got, "velocityverlet")


def test_steps_of_several_launches(gpu_lib):
    """More steps without a half-list build than one launch takes."""
    w = wl.make_workload(5, sigma=0.05, temperature=300.0, ivol=0, press_gpa=1.0, nbrupdate=5000, seed=4)
    want = _steps(w, "mixed", 0.0, [1100])
    _same(want, _steps(w, "mixed", 0.0, [1, 511, 400, 188]), "split")
