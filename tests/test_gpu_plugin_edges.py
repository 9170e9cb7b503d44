"""The waveform and response kernels at the edges of their blocks (128 bins) and
of the model (dead modes, bins above the cut, geocentric angles), against the
oracle; and containers that are not one block."""

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

from tests.helpers import config0_theta  # noqa: E402


@pytest.mark.parametrize("n", [1, 127, 128, 129, 1000])
@pytest.mark.parametrize("geo", [False, True])
def test_modes_and_response(cuda_lib, oracle, n, geo):
    from pespace_gb300 import _lib
    from pespace_gb300.detector.orbit import KaplerianHeliocentric, KeplerianGeocentric
    from pespace_gb300.waveform import IMRPhenomD, IMRPhenomHM

    th = config0_theta(3.0e6)
    th[1], th[2], th[3] = 3.3, 0.7, -0.6
    freqs = np.linspace(1e-4, 0.05, n) if n > 1 else np.array([3e-3])  # past every mode's cut
    arm = np.sqrt(3.0) * 1e8 if geo else 2.5e9
    orb = KeplerianGeocentric(arm) if geo else KaplerianHeliocentric(arm, 0.0, -np.pi / 9)
    desc = oracle.geocentric(arm) if geo else oracle.heliocentric(arm, 0.0, -np.pi / 9)
    th0 = th.copy()
    th0[10] = 0.0
    hp, hc, tf, _, _, _ = oracle.phenomhm(th0, freqs, 1e-4)
    out = IMRPhenomHM(freqs, 1e-4).from_theta(th)
    one = IMRPhenomD(freqs, 1e-4).from_theta(th)
    got = [torch.stack([m[f] for m in out.values()]).cpu().numpy() for f in ("plus", "cross", "tf")]
    scale = np.abs(hp).max(axis=1, keepdims=True) + np.abs(hc).max(axis=1, keepdims=True) + 1e-300
    assert np.array_equal(np.abs(got[0]) > 0, np.abs(hp) > 0)
    assert np.max(np.abs(got[0] - hp) / scale) < 1e-10 and np.max(np.abs(got[1] - hc) / scale) < 1e-10
    assert np.max(np.abs(got[2] - tf)) <= 1e-10 * (np.abs(tf).max() + 1.0)
    ohp, ohc, otf, _ = oracle.phenomd(th0, freqs, 1e-4)
    assert np.max(np.abs(one["plus"].cpu().numpy() - ohp)) <= 1e-10 * np.abs(ohp).max()
    assert np.max(np.abs(one["cross"].cpu().numpy() - ohc)) <= 1e-10 * np.abs(ohc).max()
    assert np.max(np.abs(one["tf"].cpu().numpy() - otf)) <= 1e-10 * (np.abs(otf).max() + 1.0)
    lam, beta, psi, tc = 1.3, 1.9, 0.9, th[10]  # a latitude past the pole: cos(beta) < 0
    want = oracle.response_links(desc, freqs, hp, hc, tf, lam, beta, psi, tc)
    d = [torch.as_tensor(x, device="cuda").contiguous() for x in (freqs, hp, hc, tf)]
    links = torch.empty((6, n), dtype=torch.complex128, device="cuda")
    _lib.check(_lib.load().pes_response_links(orb.to_c(), _lib.ptr(d[0]), n, 6, _lib.ptr(d[1]), _lib.ptr(d[2]),
                                              _lib.ptr(d[3]), lam, beta, psi, tc, _lib.ptr(links), _lib.stream_handle()))
    norm = np.sum(np.abs(want), axis=0) + 1e-300
    assert np.max(np.abs(links.cpu().numpy() - want) / norm) < 1e-13


def test_stacked_containers(cuda_lib):
    from pespace_gb300.detector.antenna import _stacked
    from pespace_gb300.inference.likelihood import _rows

    block = torch.randn(3, 8, dtype=torch.complex128, device="cuda")
    for rows in ([block[0], block[1], block[2]], [block[2], block[0], block[1]], [block[0], block[0], block[1]],
                 [block[k].conj() for k in range(3)], [block[0].conj()], [block[k, ::2] for k in range(3)],
                 [block[0], block[1].clone(), block[2]]):
        got = _stacked(rows, torch.complex128)
        assert got.is_contiguous() and not got.is_conj() and torch.equal(got, torch.stack(rows).resolve_conj())
    assert _stacked([block[0], block[1], block[2]], torch.complex128).data_ptr() == block.data_ptr()
    for data in (block, block.conj(), block[:, ::2]):
        for ch in (("A", "E", "T"), ("T", "A"), ("E",)):
            got = _rows(data, ("A", "E", "T"), ch)
            assert got.is_contiguous() and not got.is_conj()
            assert torch.equal(got, data[["AET".index(c) for c in ch]].resolve_conj())
