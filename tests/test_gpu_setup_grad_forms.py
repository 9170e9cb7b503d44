"""The mixed gradient's set-up has two forms, by groups of lanes up to 192 samples and
by one thread per sample beyond: the same gradients from both (up to the order of
the FP32 moment atomics), and those of the oracle (the mixed gradient's bar, 1e-3)."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

from tests.helpers import config0_theta, make_dataset, perturbed, random_prior_theta  # noqa: E402
from tests.test_gpu_plan import cuda_detectors, lisa  # noqa: E402

GRID = (2.0 ** 16, 8.0, 1e-4, 0.03)


def test_both_sides_of_the_rule(cuda_lib, oracle):
    from pespace_gb300.inference import WhittleLikelihood

    th0 = config0_theta(GRID[0] - 8000.0)
    g, dets = make_dataset(oracle, *GRID, [lisa(oracle)], th0, seed=5)
    eng = WhittleLikelihood(cuda_detectors(g, dets, GRID), precision="mixed", reference_frequency=1e-4, cut_factor=1.2,
                            max_batch=193)
    rng = np.random.default_rng(6)
    thetas = np.concatenate([th0[None], [perturbed(th0, rng) for _ in range(95)], random_prior_theta(rng, 97, th0[10])])
    thetas[17, 1] = 0.5  # outside the domain
    l1, g1 = eng.log_likelihood_and_grad(thetas[:192])
    l2, g2 = eng.log_likelihood_and_grad(thetas)
    assert torch.equal(l1, l2[:192])
    norm = torch.linalg.norm(g1, dim=1, keepdim=True)
    norm[17] = 1.0
    assert torch.max(torch.abs(g2[:192] - g1) / norm).item() < 1e-5
    rows = [0, 5, 60, 192]
    want = oracle.Plan(g, [(o, k, d, p) for _, o, k, d, p in dets], 1e-4, cut_factor=1.2).lnl(thetas[rows], grad=True)[1]
    scale = np.linalg.norm(want, axis=1, keepdims=True)
    assert np.max(np.abs(g2.cpu().numpy()[rows] - want) / scale) < 1e-3
