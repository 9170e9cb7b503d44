"""Float-float time-domain TDI where a window's links differ by up to 2^90: a channel
that reads only the small ones keeps their 48 bits (X, Y, Z on their own; Z reads
neither link 12 nor 21), down to the level at which floats flush: 2^-126 of the
window's largest sample, each of a channel's terms and the output's tail."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

from oracle import td_tdi  # noqa: E402
from tests.test_td_tdi import LISA_ARM_SEC, MIXED_TOL, _run_gpu  # noqa: E402


@pytest.mark.parametrize("gen", ["1.5", "2.0"])
@pytest.mark.parametrize("bits", [0, 40, 73, 80, 90])
def test_small_links(cuda_lib, gen, bits):
    n, dt = 3000, 5.0
    added = td_tdi.layout(LISA_ARM_SEC, dt, gen)[0]
    links = np.random.default_rng(bits).uniform(1.0, 2.0, (1, 6, n + added)) * 1e-21
    links[:, 2:] *= 2.0 ** -bits  # links 12 and 21 are the first two
    got = _run_gpu(links, n, LISA_ARM_SEC, dt, gen, False, mixed=True)[0]
    want = td_tdi.combine(links[0], n, LISA_ARM_SEC, dt, gen, False)
    assert np.max(np.abs(got[:2] - want[:2])) <= MIXED_TOL * 2e-21
    flush = (2 if gen == "1.5" else 4) * 4 + 1
    assert np.max(np.abs(got[2] - want[2])) <= 2e-21 * (MIXED_TOL * 2.0 ** -bits + flush * 2.0 ** -126)
