"""FP64 plans have no launch that ``sample_threads`` reaches: the autotuner times
them once and leaves the option as it was."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from tests.helpers import config0_theta, make_dataset  # noqa: E402
from tests.test_gpu_plan import DT, DUR, FMAX, FMIN, cuda_detectors, lisa  # noqa: E402


@pytest.mark.parametrize("value", [8, 32])
def test_one_candidate(cuda_lib, oracle, value):
    from pespace_gb300.inference import WhittleLikelihood
    from pespace_gb300.inference.autotune import set_option

    th0 = config0_theta(DUR - 20000.0)
    g, dets = make_dataset(oracle, DUR, DT, FMIN, FMAX, [lisa(oracle)], th0)
    eng = WhittleLikelihood(cuda_detectors(g, dets), precision="fp64", reference_frequency=1e-4, max_batch=2)
    set_option(eng, "sample_threads", value)
    report = eng.autotune(np.stack([th0, th0]), grad=False, reps=1)
    assert list(report) == ["sample_threads"] and report["sample_threads"]["chosen"] == value
    assert list(report["sample_threads"]["ms"]) == [value] and eng.launch_options["sample_threads"] == value
