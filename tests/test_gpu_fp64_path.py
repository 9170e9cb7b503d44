"""The dense FP64 pass of IMRPhenomD plans where its branches change: both bin
counts per thread (small and large calls), blocks with one live bin, geocentric
and heliocentric detectors, bands whose sin(x)/x arguments leave the short and
then every Taylor series, both TDI generations, channel subsets.

Bars: lnL and gradient of the FP64 plan against the oracle, as for the plan
(1e-6 + 1e-11 relative, 1e-7 of the gradient norm)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from tests.helpers import config0_theta, make_dataset, random_prior_theta  # noqa: E402
from tests.test_gpu_mixed import taiji  # noqa: E402
from tests.test_gpu_plan import cuda_detectors, lisa, tianqin  # noqa: E402


@pytest.mark.parametrize("grid,gen,kinds,batch,chans", [
    ((2.0 ** 16, 8.0, 1e-4, 0.03), "1.5", "LT", 3, "AET"),      # small call: one bin per thread
    ((2.0 ** 18, 8.0, 1e-4, 0.03), "2.0", "L", 40, "AET"),      # 2 480 blocks of 128 bins: four bins per thread
    ((2.0 ** 15, 4.0, 1e-3, 0.12), "1.5", "JT", 4, "AET"),      # Taiji beyond f L = 1: arguments up to 7.5
    ((129 * 64.0, 4.0, 1e-2, 0.0257), "1.5", "L", 2, "AE"),     # 129 bins: a block with one bin
    ((2.0 ** 15, 8.0, 1e-4, 0.02), "2.0", "LJT", 2, "T"),
])
def test_fp64_lnl_and_gradient_against_oracle(cuda_lib, oracle, grid, gen, kinds, batch, chans):
    from pespace_gb300.inference import WhittleLikelihood

    th0 = config0_theta(grid[0] * 0.9)
    make = {"L": lisa, "J": taiji, "T": tianqin}
    g, dets = make_dataset(oracle, *grid, [make[k](oracle, gen) for k in kinds], th0, seed=9)
    eng = WhittleLikelihood(cuda_detectors(g, dets, grid), channels=tuple(chans), precision="fp64",
                            reference_frequency=1e-4, cut_factor=1.2 if batch == 40 else 0.0, max_batch=batch)
    thetas = np.concatenate([th0[None], random_prior_theta(np.random.default_rng(batch), batch - 1, th0[10])])
    thetas[-1, 5], thetas[-1, 7] = -1.0, 0.0  # face on, in the ecliptic
    plan = oracle.Plan(g, [(o, k, d, p) for _, o, k, d, p in dets], 1e-4, channels=tuple(chans),
                       cut_factor=1.2 if batch == 40 else 0.0)
    want, want_grad = plan.lnl(thetas, grad=True, nthreads=8)
    lnl, grad = eng.log_likelihood_and_grad(thetas)
    only = eng.log_likelihood_batch(thetas).cpu().numpy()
    for got in (lnl.cpu().numpy(), only):
        assert np.all(np.abs(got - want) <= 1e-6 + 1e-11 * np.abs(want)), got - want
    norm = np.linalg.norm(want_grad, axis=1, keepdims=True)
    assert np.max(np.abs(grad.cpu().numpy() - want_grad) / norm) < 1e-7
