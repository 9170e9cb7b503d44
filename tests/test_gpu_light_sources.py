"""Light sources decades before they merge: phases past 2^45 rad, where the FP64
path's table sine and cosine no longer reduce their argument.  Such a phase has no
correct digits, but its sine and cosine are a point of the unit circle: amplitudes,
and lnL on data without a signal, which is -<h|h>/2, do not depend on it."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

from tests.helpers import config0_theta, make_dataset  # noqa: E402
from tests.test_gpu_plan import cuda_detectors, lisa, tianqin  # noqa: E402

GRID = (2.0 ** 18, 8.0, 1e-5, 0.03)


def light(mtot):
    th = config0_theta(GRID[0] * 0.9)
    th[0], th[1] = np.log(mtot * 0.25 ** 0.6), 1.0
    th[4] = np.log(1e-3)
    return th


@pytest.mark.parametrize("mtot", [0.003, 0.3, 30.0])
def test_waveforms(cuda_lib, oracle, mtot):
    from pespace_gb300.waveform import IMRPhenomD, IMRPhenomHM

    freqs = np.geomspace(1e-5, 0.05, 300)
    th = light(mtot)
    th0 = th.copy()
    th0[10] = 0.0
    hp, hc, _, _ = oracle.phenomd(th0, freqs, 1e-4)
    one = IMRPhenomD(freqs, 1e-4).from_theta(th)
    for got, want in ((one["plus"], hp), (one["cross"], hc)):
        assert np.max(np.abs(np.abs(got.cpu().numpy()) / np.abs(want) - 1.0)) < 1e-10
    hp, hc, _, _, _, _ = oracle.phenomhm(th0, freqs, 1e-4)
    for k, m in enumerate(IMRPhenomHM(freqs, 1e-4).from_theta(th).values()):
        got = np.abs(m["plus"].cpu().numpy())
        assert np.max(np.abs(got - np.abs(hp[k])) / (np.abs(hp[0]) + np.abs(hc[0]))) < 1e-10


@pytest.mark.parametrize("mtot", [0.003, 0.3])
def test_response_and_tdi_of_any_argument(cuda_lib, oracle, mtot):
    """Times of 1e20 s and more: the links stay bounded by the pattern's largest value (2 a |h|)."""
    from pespace_gb300 import _lib
    from pespace_gb300.detector.orbit import KaplerianHeliocentric

    n = 200
    freqs = np.geomspace(1e-5, 0.05, n)
    hp, hc, tf, _ = oracle.phenomd(light(mtot), freqs, 1e-4)
    for tc in (0.0, 1e21):
        d = [torch.as_tensor(x[None] if x.ndim == 1 and k else x, device="cuda").contiguous()
             for k, x in enumerate((freqs, hp, hc, -1e3 * np.abs(tf)))]
        links = torch.empty((6, n), dtype=torch.complex128, device="cuda")
        _lib.check(_lib.load().pes_response_links(KaplerianHeliocentric(2.5e9, 0.0, -np.pi / 9).to_c(), _lib.ptr(d[0]),
                                                  n, 1, _lib.ptr(d[1]), _lib.ptr(d[2]), _lib.ptr(d[3]), 1.3, 0.4, 0.9,
                                                  tc, _lib.ptr(links), _lib.stream_handle()))
        bound = 2.0 * np.pi * freqs * (2.5e9 / 299792458.0) * (np.abs(hp) + np.abs(hc))
        assert np.all(np.abs(links.cpu().numpy()) <= bound)


@pytest.mark.parametrize("mtot", [0.003, 0.3])
def test_fp64_plan(cuda_lib, oracle, mtot):
    from pespace_gb300.inference import WhittleLikelihood

    th = light(mtot)
    g, dets = make_dataset(oracle, *GRID, [lisa(oracle), tianqin(oracle)], th, seed=9)
    for d in dets:
        d[3] = np.zeros_like(d[3])
    eng = WhittleLikelihood(cuda_detectors(g, dets, GRID), precision="fp64", reference_frequency=1e-4, max_batch=1)
    want = oracle.Plan(g, [(o, k, d, p) for _, o, k, d, p in dets], 1e-4).lnl(th[None])
    lnl, grad = eng.log_likelihood_and_grad(th)
    # at 3 mHz, where the sum lies, t(f) is 2e17 s and TianQin's angle 4e12 rad, which
    # carries a rounding of 1e-3 rad: |h|^2 of a bin by twice that, in either code
    for got in (lnl, eng.log_likelihood_batch(th)):
        assert abs(float(got[0]) / float(want[0]) - 1.0) < 5e-3
    assert bool(torch.isfinite(grad).all())
    assert abs(float(grad[0, 4]) / (-2.0 * float(lnl[0])) - 1.0) < 1e-9  # d lnL / d ln D_L = <h|h>
