"""Knots of a batched fit that the tables do not show: the gradient of a knot
whose amplitude is zero, against the single-system path (1e-8 of its norm, as
for every knot)."""
import numpy as np
import pytest
import torch

from moldy_b200 import MoldySystem
from moldy_b200 import adjoint as adj
from moldy_b200.potentials import FE_FE
from tests.test_gpu_adjoint import fm_config, gpu_eval

pytestmark = pytest.mark.gpu


def test_batch_gradient_of_a_knot_without_amplitude(gpu_lib):
    """A pair knot past every other with amplitude zero, as a fit starts a new
    one: the tables end before it, its gradient comes from the pairs between
    (the single-system path walks the half list and has them)."""
    from moldy_b200 import MoldyBatch
    w = fm_config(91, n=6, sigma=0.12)
    base = {k: np.asarray(getattr(FE_FE, k), dtype=np.float64) for k in adj.KNOT_NAMES}
    base["av"] = np.concatenate([[0.0, 0.0], base["av"]])
    base["rv"] = np.concatenate([[4.9, 4.3], base["rv"]])
    s = MoldySystem.from_workload(w, uselookup=True)
    _, f0, s0 = gpu_eval(s, coeffs=FE_FE)
    ref = (f0 + 1e-2 * np.random.default_rng(3).normal(size=f0.shape), s0 * 1.1)
    th1 = {k: torch.tensor(v, requires_grad=True) for k, v in base.items()}
    adj.force_matching_knots([s], [(w.x0, w.b0)], [ref], th1).backward()
    s.close()
    b = MoldyBatch.from_workloads([w])
    b.set_references([ref[0]], [ref[1]])
    th2 = {k: torch.tensor(v, requires_grad=True) for k, v in base.items()}
    adj.batch_force_matching_knots(b, th2).backward()
    b.close()
    for k in adj.KNOT_NAMES:
        a, g = th1[k].grad.numpy(), th2[k].grad.numpy()
        assert np.max(np.abs(a - g)) <= 1e-8 * np.linalg.norm(a), (k, a, g)
    assert np.all(np.abs(th1["av"].grad.numpy()[:2]) > 0.0)
