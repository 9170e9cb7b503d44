"""Per-sample set-up by groups of lanes: two samples share each warp, so a
sample's result must not depend on its neighbours, on the batch's remainder or
on a neighbour outside the parameter domain."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

from tests.helpers import config0_theta, make_dataset, random_prior_theta  # noqa: E402
from tests.test_gpu_plan import cuda_detectors, lisa, tianqin  # noqa: E402

GRID = (2.0 ** 16, 8.0, 1e-4, 0.03)


@pytest.mark.parametrize("precision,approximant", [("fp64", "IMRPhenomD"), ("mixed", "IMRPhenomD"),
                                                   ("fp64", "IMRPhenomHM"), ("mixed", "IMRPhenomHM")])
@pytest.mark.parametrize("batch", [1, 2, 5])
def test_samples_do_not_depend_on_their_neighbours(cuda_lib, oracle, precision, approximant, batch):
    from pespace_gb300.inference import WhittleLikelihood

    th0 = config0_theta(GRID[0] - 8000.0)
    g, dets = make_dataset(oracle, *GRID, [lisa(oracle), tianqin(oracle)], th0, seed=5)
    eng = WhittleLikelihood(cuda_detectors(g, dets, GRID), precision=precision, reference_frequency=1e-4,
                            cut_factor=1.2, max_batch=8, n_sparse=256, approximant=approximant)
    thetas = random_prior_theta(np.random.default_rng(batch), batch, th0[10])
    got = eng.log_likelihood_batch(thetas)
    fisher = eng.fisher_matrix(thetas)
    bad = np.repeat(thetas, 2, axis=0)[: 2 * batch]
    bad[1::2, 1] = 0.5  # every sample beside one outside the domain
    for lo in range(0, batch, 4):
        part = eng.log_likelihood_batch(bad[2 * lo:2 * lo + 8])
        assert torch.equal(part[::2], got[lo:lo + 4]) and bool(torch.isneginf(part[1::2]).all())
    for k in range(batch):
        assert torch.equal(eng.log_likelihood_batch(thetas[k]), got[k:k + 1])
        assert torch.equal(eng.fisher_matrix(thetas[k])[0], fisher[k])
    if approximant == "IMRPhenomD" or precision == "fp64":
        lnl, grad = eng.log_likelihood_and_grad(thetas)
        for k in range(batch):
            l1, g1 = eng.log_likelihood_and_grad(thetas[k])
            assert torch.equal(l1[0], lnl[k])
            assert torch.max(torch.abs(g1[0] - grad[k])) <= 1e-5 * torch.linalg.norm(grad[k])
