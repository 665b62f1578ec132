"""What a batch refuses stays refused, and what it goes on with is sound: a cut
too long for a box, boxes too narrow for the cut, in any order of calls."""
import dataclasses

import numpy as np
import pytest

from moldy_b200 import MoldyBatch
from moldy_b200 import workloads as wl
from moldy_b200._lib import MoldyError

pytestmark = pytest.mark.gpu


def _batch():
    ws = [wl.make_workload(n, sigma=0.1, temperature=0.0, ivol=1, seed=n) for n in (4, 5)]
    b = MoldyBatch.from_workloads(ws)
    return ws, b, b.force(), b.forces()


def _stretched(c, factor):
    """The same functions with every knot of the pair function moved out."""
    return dataclasses.replace(c, rv=np.asarray(c.rv) * factor)


def _same(b, out, f):
    got = b.force()
    assert all(np.array_equal(got[k], out[k]) for k in out)
    assert np.array_equal(b.forces(), f)


def test_cut_too_long_is_refused_every_time(gpu_lib):
    ws, b, out, f = _batch()
    long = _stretched(ws[0].coeffs, 1.8)
    for _ in range(2):
        with pytest.raises(MoldyError, match="narrower than twice"):
            b.set_up_fetm(long)
        with pytest.raises(MoldyError, match="do not cover"):
            b.force()
    b.set_up_fetm(ws[0].coeffs)
    _same(b, out, f)
    b.close()


def test_narrow_boxes_are_refused_every_time(gpu_lib):
    ws, b, out, f = _batch()
    narrow = [0.5 * w.b0 for w in ws]
    for _ in range(2):
        with pytest.raises(MoldyError, match="narrower than twice"):
            b.set_state(b0=narrow)
        with pytest.raises(MoldyError, match="narrower than twice"):
            b.set_up_fetm(ws[0].coeffs)
    _same(b, out, f)                     # the boxes on the device are the old ones
    flat = [w.b0.copy() for w in ws]
    flat[1][:, 2] = flat[1][:, 1]
    with pytest.raises(MoldyError, match="singular"):
        b.set_state(b0=flat)
    b.set_state(b0=[w.b0 for w in ws])
    _same(b, out, f)
    with pytest.raises(MoldyError, match="singular"):
        b.set_state(b0=flat)
    b.set_skin(0.3)                      # lays the last accepted boxes out again
    _same(b, out, f)
    b.close()
