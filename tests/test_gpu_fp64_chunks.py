"""The FP64 IMRPhenomD plan's block partials: the gradient of many samples runs in
chunks of what the workspace holds, bit for bit as the samples of smaller calls,
and the workspace grows with max_batch by five doubles per 512 bins and sample."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

from tests.helpers import config0_theta, make_dataset, random_prior_theta  # noqa: E402
from tests.test_gpu_plan import cuda_detectors, lisa  # noqa: E402


def _engine(oracle, grid, max_batch, th0):
    from pespace_gb300.inference import WhittleLikelihood

    g, dets = make_dataset(oracle, *grid, [lisa(oracle)], th0, seed=9)
    det = cuda_detectors(g, dets, grid)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    eng = WhittleLikelihood(det, precision="fp64", reference_frequency=1e-4, max_batch=max_batch)
    return eng, free - torch.cuda.mem_get_info()[0], g["freqs"].size


def test_gradient_in_chunks(cuda_lib, oracle):
    grid = (2.0 ** 20, 8.0, 1e-4, 0.03)  # 62 blocks of 512 bins: chunks of 264 samples
    th0 = config0_theta(grid[0] * 0.9)
    eng, _, _ = _engine(oracle, grid, 300, th0)
    thetas = np.concatenate([th0[None], random_prior_theta(np.random.default_rng(3), 299, th0[10])])
    thetas[265, 1] = 0.5  # outside the domain, in the second chunk
    lnl, grad = eng.log_likelihood_and_grad(thetas)
    status = eng.last_status.clone()
    assert bool(torch.isneginf(lnl[265])) and not bool(grad[265].any())
    for lo, hi in ((0, 40), (250, 290), (263, 300)):
        l1, g1 = eng.log_likelihood_and_grad(thetas[lo:hi])
        assert torch.equal(l1, lnl[lo:hi]) and torch.equal(g1, grad[lo:hi])
        assert torch.equal(eng.last_status, status[lo:hi])


def test_workspace_per_sample(cuda_lib, oracle):
    grid = (2.0 ** 22, 8.0, 1e-4, 0.03)
    th0 = config0_theta(grid[0] * 0.9)
    one, small, n = _engine(oracle, grid, 1, th0)
    batch = 2048
    many, large, _ = _engine(oracle, grid, batch, th0)
    # five doubles per block of 512 bins, 16 KB of set-up blocks per sample, 16 MB of the allocator's rounding
    assert large - small <= batch * (40 * (-(-n // 512)) + 16384) + (16 << 20)
    del one, many
