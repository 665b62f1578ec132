"""A batch whose rows of the pairs inside the cut find no memory, or give it up
for a buffer that is needed more, does without them: the FP64 passes walk the
list rows, the persistent evaluation leaves the batch to the per-pass form.

Tolerances: a quench adds row by row either way, so its results are the same
bits; the other FP64 sums are grouped by lanes over other rows, 1e-12; the
mixed per-pass form is the same code either way.
"""
import numpy as np
import pytest

from moldy_b200 import MoldyBatch
from moldy_b200 import workloads as wl
from tests.helpers import rel_norm_err

pytestmark = pytest.mark.gpu
SIZES = [14, 9, 16, 5] * 20       # 307,760 atoms: rows of 59 MB


def _batch():
    rng = np.random.default_rng(5)
    ws = [wl.make_workload(n, sigma=0.08, temperature=0.0, ivol=1, seed=k, strain=wl.random_symmetric_strain(rng, 0.02))
          for k, n in enumerate(SIZES)]
    return MoldyBatch.from_workloads(ws)


def _evaluate(b, per_pass):
    out = {}
    r = b.force()
    out["force"] = [r["pe"], r["tp"], b.forces(), b.density()["rho"], np.concatenate(b.energies())]
    loss, grads = b.force_matching()
    out["fit"] = [loss] + [grads[k] for k in ("dvee", "phi", "dphi", "demb")]
    b.set_precision("mixed")
    b.set_energy_calc(False)
    b.set_persistent(not per_pass)
    r = b.force()
    out["mixed"] = [r["pe"], r["tp"], b.forces()]
    b.set_precision("fp64")
    b.set_energy_calc(True)
    q = b.quench(maxfn=6)
    out["quench"] = [np.asarray(q[k]) for k in sorted(q)] + [b.get_state()]
    return out


def _fill(torch, leave):
    torch.cuda.synchronize()
    fill = torch.empty(torch.cuda.mem_get_info()[0] - leave, dtype=torch.uint8, device="cuda")
    assert torch.cuda.mem_get_info()[0] <= leave + (4 << 20)
    return fill


@pytest.fixture(scope="module")
def with_rows(gpu_lib):
    import torch
    nt = sum(2 * n ** 3 for n in SIZES)
    rng = np.random.default_rng(1)
    refs = (rng.normal(size=(nt, 3)) * 0.1, rng.normal(size=(len(SIZES), 3, 3)) * 0.01)
    torch.zeros(1, device="cuda")
    _batch().close()
    free = torch.cuda.mem_get_info()[0]
    b = _batch()
    b.set_references(*refs)
    b.force_matching()
    used = free - torch.cuda.mem_get_info()[0]
    out = _evaluate(b, per_pass=True)
    b.close()
    assert 48 * 4 * nt > 56 << 20
    return refs, used, out


@pytest.mark.parametrize("when", ["at creation", "for the references"])
def test_batch_without_memory_for_the_inside_rows(with_rows, when):
    import torch
    refs, used, want = with_rows
    if when == "at creation":
        fill = _fill(torch, used - (40 << 20))
        b = _batch()
    else:
        b = _batch()
        fill = _fill(torch, 8 << 20)
    b.set_references(*refs)
    got = _evaluate(b, per_pass=False)
    del fill
    torch.cuda.empty_cache()
    b.close()
    for k in ("quench", "mixed"):
        for p, q in zip(got[k], want[k]):
            assert np.array_equal(p, q), k
    for k in ("force", "fit"):
        for p, q in zip(got[k], want[k]):
            assert rel_norm_err(p, q) < 1e-12, k
