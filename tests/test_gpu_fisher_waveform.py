"""Mixed Fisher matrices where the waveform's tangents are hardest: unequal masses,
high spins and heavy sources whose merger-ringdown fills the band, against the
FP64 plan (the mixed plan's bar, 1e-5); and the first call of a plan under a
relaxed stream capture."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

from tests.helpers import config0_theta, make_dataset  # noqa: E402
from tests.test_gpu_fisher import _normalised_err  # noqa: E402
from tests.test_gpu_plan import cuda_detectors, lisa  # noqa: E402

GRID = (2.0 ** 18, 8.0, 1e-4, 0.03)


def _engine(oracle, precision, th0, max_batch):
    from pespace_gb300.inference import WhittleLikelihood

    g, dets = make_dataset(oracle, *GRID, [lisa(oracle)], th0, seed=4)
    return WhittleLikelihood(cuda_detectors(g, dets, GRID), precision=precision, reference_frequency=1e-4,
                             max_batch=max_batch)


@pytest.mark.parametrize("q", [1.0, 5.0, 8.0])
@pytest.mark.parametrize("mtot", [2e5, 2e6, 2e7])
def test_unequal_masses_and_high_spins(cuda_lib, oracle, q, mtot):
    th0 = config0_theta(GRID[0] - 20000.0)
    rows = []
    for chi1, chi2 in ((0.95, 0.9), (-0.95, 0.8), (0.0, -0.95)):
        th = th0.copy()
        th[0] = np.log(mtot * (q / (1 + q) ** 2) ** 0.6)
        th[1:4] = q, chi1, chi2
        rows.append(th)
    thetas = np.stack(rows)
    got = _engine(oracle, "mixed", th0, 3).fisher_matrix(thetas).cpu().numpy()
    want = _engine(oracle, "fp64", th0, 3).fisher_matrix(thetas).cpu().numpy()
    assert _normalised_err(got, want) < 1e-5


@pytest.mark.parametrize("precision", ["mixed", "fp64"])
def test_first_call_under_relaxed_capture(cuda_lib, oracle, precision):
    """The first call allocates and fills its tables; a relaxed capture permits that."""
    th0 = config0_theta(GRID[0] - 20000.0)
    eng = _engine(oracle, precision, th0, 2)
    theta = torch.as_tensor(np.stack([th0, th0]), device="cuda")
    theta[1, 0] += 0.5
    graph = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(graph, capture_error_mode="relaxed"):
        out = eng.fisher_matrix(theta)
    graph.replay()
    torch.cuda.synchronize()
    captured = out.clone()
    assert torch.equal(captured, eng.fisher_matrix(theta)) and bool(torch.isfinite(captured).all())
