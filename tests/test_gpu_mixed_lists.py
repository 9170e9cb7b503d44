"""The mixed plan's re-evaluation lists, exact ranges and final sums: a sample's
lnL does not depend on the batch it is in (sizes about the four samples of a
block of the final sums, samples listed and not, outside the domain, detectors
with different exact ranges)."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

from tests.helpers import config0_theta, make_dataset, perturbed  # noqa: E402
from tests.test_gpu_mixed import taiji  # noqa: E402
from tests.test_gpu_plan import DT, DUR, FMAX, FMIN, cuda_detectors, lisa  # noqa: E402


@pytest.mark.parametrize("approximant", ["IMRPhenomD", "IMRPhenomHM"])
@pytest.mark.parametrize("refine_all", [False, True])
def test_batch_independent(cuda_lib, oracle, approximant, refine_all):
    from pespace_gb300.inference import WhittleLikelihood

    th0 = config0_theta(DUR - 20000.0)
    g, dets = make_dataset(oracle, DUR, DT, FMIN, FMAX, [lisa(oracle), taiji(oracle)], th0, seed=4)
    rng = np.random.default_rng(5)
    thetas = np.stack([th0] + [perturbed(th0, rng) for _ in range(8)])
    thetas[3, 0] += 1.5  # a heavier source: a short range
    thetas[5, 1] = 0.5   # outside the domain
    thetas[6, 4] -= 2.0  # louder
    eng = WhittleLikelihood(cuda_detectors(g, dets), precision="mixed", reference_frequency=1e-4, cut_factor=1.2,
                            max_batch=9, approximant=approximant)
    eng.refine_all = refine_all
    single = torch.cat([eng.log_likelihood_batch(thetas[k:k + 1]) for k in range(9)]).cpu().numpy()
    assert np.isneginf(single[5]) and np.isfinite(np.delete(single, 5)).all()
    for n in (3, 4, 5, 9):
        got = eng.log_likelihood_batch(thetas[:n]).cpu().numpy()
        assert np.array_equal(got, single[:n]), (n, got - single[:n])
