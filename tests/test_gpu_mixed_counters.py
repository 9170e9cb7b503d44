"""The mixed plan's re-evaluation lists start empty in every call, however few
threads its one-thread-per-sample launches have: one sample at one thread per
block, listed call after call, gives what it gives with the default option."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

from tests.helpers import config0_theta, make_dataset  # noqa: E402
from tests.test_gpu_plan import DT, DUR, FMAX, FMIN, cuda_detectors, lisa  # noqa: E402


@pytest.mark.parametrize("approximant", ["IMRPhenomD", "IMRPhenomHM"])
@pytest.mark.parametrize("max_batch", [1, 3])
def test_one_sample_with_one_thread(cuda_lib, oracle, approximant, max_batch):
    from pespace_gb300.inference import WhittleLikelihood
    from pespace_gb300.inference.autotune import set_option

    th0 = config0_theta(DUR - 20000.0)
    g, dets = make_dataset(oracle, DUR, DT, FMIN, FMAX, [lisa(oracle)], th0, seed=4)
    eng = WhittleLikelihood(cuda_detectors(g, dets), precision="mixed", reference_frequency=1e-4, cut_factor=1.2,
                            max_batch=max_batch, approximant=approximant)
    eng.refine_all = True
    loud = th0.copy()
    loud[4] -= 4.0  # its splines' error estimate asks for the exact re-evaluation
    for theta in (th0, loud):
        set_option(eng, "sample_threads", 8)
        want = eng.log_likelihood_batch(theta)
        kinds = eng.last_work(1)
        assert kinds["refined_ff"] + kinds["refined_exact"] == 1
        set_option(eng, "sample_threads", 1)
        for _ in range(4):
            assert torch.equal(eng.log_likelihood_batch(theta), want)
            assert eng.last_work(1) == kinds
        if approximant == "IMRPhenomD":
            set_option(eng, "sample_threads", 8)
            lnl, grad = eng.log_likelihood_and_grad(theta)
            set_option(eng, "sample_threads", 1)
            for _ in range(2):
                l1, g1 = eng.log_likelihood_and_grad(theta)
                assert torch.equal(l1, lnl) and torch.equal(l1, want)
                # the order of the gradient's FP32 moment atomics
                assert torch.max(torch.abs(g1 - grad)).item() <= 1e-5 * float(np.linalg.norm(grad.cpu().numpy()))
