"""Mixed Fisher matrices at the edges of their groups of 128 bins (pairs of
groups per block, the summing warps' last group, a sample cut inside the band),
on two detectors, against the oracle's FP64 dual-number matrices (the mixed
plan's bar, 1e-5).  The bands start at 3 mHz: at the lowest frequencies the T
channel is a cancellation of the links that FP32 does not resolve."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from tests.helpers import config0_theta, make_dataset, perturbed  # noqa: E402
from tests.test_gpu_fisher import _normalised_err  # noqa: E402
from tests.test_gpu_plan import DT, DUR, cuda_detectors, lisa  # noqa: E402
from tests.test_gpu_mixed import taiji  # noqa: E402


@pytest.mark.parametrize("bins", [127, 128, 129, 255, 257, 1025, 5000])
@pytest.mark.parametrize("batch", [1, 3])
def test_fisher_group_edges(cuda_lib, oracle, bins, batch):
    from pespace_gb300.inference import WhittleLikelihood

    fmin = 3e-3
    fmax = fmin + (bins - 0.5) / (DT * (DUR // DT + 1))
    th0 = config0_theta(DUR - 20000.0)
    g, dets = make_dataset(oracle, DUR, DT, fmin, fmax, [lisa(oracle), taiji(oracle)], th0, seed=4)
    assert abs(g["freqs"].size - bins) <= 1
    rng = np.random.default_rng(bins)
    thetas = np.stack([th0] + [perturbed(th0, rng) for _ in range(batch - 1)])
    if batch > 1:
        thetas[1, 0] += 1.0  # heavier: its cut falls inside the longest band
    eng = WhittleLikelihood(cuda_detectors(g, dets, (DUR, DT, fmin, fmax)), precision="mixed", reference_frequency=1e-4, cut_factor=1.2,
                            max_batch=batch)
    got = eng.fisher_matrix(thetas).cpu().numpy()
    want = oracle.Plan(g, [(o, gen, d, p) for _, o, gen, d, p in dets], 1e-4, cut_factor=1.2).fisher(thetas)
    assert np.array_equal(got, np.swapaxes(got, 1, 2))
    assert _normalised_err(got, want) < 1e-5
    assert np.array_equal(got, eng.fisher_matrix(thetas).cpu().numpy())
