"""Bins whose waveform is zero: their links are zero, unless an angle, a time or the
frequency is not finite, which shows in every bin."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("what", ["none", "lam", "beta", "psi", "tc", "f", "tf", "infinite tc"])
def test_zero_waveform(cuda_lib, what):
    from pespace_gb300 import _lib
    from pespace_gb300.detector.orbit import KaplerianHeliocentric

    n = 130
    bad = float("inf") if what == "infinite tc" else float("nan")
    freqs = torch.linspace(1e-4, 1e-2, n, dtype=torch.float64, device="cuda")
    h = torch.zeros((2, n), dtype=torch.complex128, device="cuda")
    tf = torch.zeros((2, n), dtype=torch.float64, device="cuda")
    angle = {"lam": 0.3, "beta": 0.2, "psi": 0.1, "tc": 5.0}
    if what in angle:
        angle[what] = bad
    elif what == "infinite tc":
        angle["tc"] = bad
    elif what == "f":
        freqs[:] = bad
    elif what == "tf":
        tf[:] = bad
    links = torch.empty((6, n), dtype=torch.complex128, device="cuda")
    _lib.check(_lib.load().pes_response_links(KaplerianHeliocentric(2.5e9, 0.0, -np.pi / 9).to_c(), _lib.ptr(freqs), n, 2,
                                              _lib.ptr(h), _lib.ptr(h), _lib.ptr(tf), angle["lam"], angle["beta"],
                                              angle["psi"], angle["tc"], _lib.ptr(links), _lib.stream_handle()))
    got = torch.view_as_real(links)
    assert bool((got == 0.0).all()) if what == "none" else bool(got.isnan().all())
