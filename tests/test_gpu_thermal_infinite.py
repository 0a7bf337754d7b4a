"""Thermal fluxes where a denominator vanishes (no beaming: an infinite temperature; a band so
long that its exponential is one): the band's own value, infinite as in the reference, and
the other bands untouched (1e-12 relative of the oracle)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BANDS = {"two": ([4700.0, 8000.0], False), "uv": ([5.0, 4602.8, 22088.3], False),
         "wise": ([3352.6, 4602.8, 11098.4, 22640.5], True), "radio": ([4700.0, 1e30, 5.0], False),
         "eight": ([9.0, 550.0, 2200.0, 3400.0, 4600.0, 12000.0, 1e30, 1e5], False)}


@pytest.mark.parametrize("name", BANDS)
def test_vanishing_denominators(gpu, oracle, name):
    bands, cc = BANDS[name]
    nb, n = len(bands), 6
    s2obj = np.repeat([[1.2], [0.3], [0.1]], n, axis=1)
    s2obs = np.repeat([[0.9], [-0.4], [0.0]], n, axis=1)
    beam = np.array([0.0, 1.1, 0.0, 1e-300, 0.9, 1e-60])
    alb = np.full((nb, n), 0.1)
    got = gpu.flux.neatm_arrays(s2obj, s2obs, np.full(n, 15.0), 0.15, np.full(n, 1.0),
                                np.full(n, 0.1), beam, 0.9, bands, alb, None, [100.0] * nb, cc)
    for i in range(n):
        want = oracle.neatm_total_flux(s2obj[:, i], s2obs[:, i], 15.0, 0.15, 1.0, 0.1, beam[i], 0.9,
                                       bands, [0.1] * nb, None, [100.0] * nb, cc)
        # a temperature of 1e15 K and more leaves exp(x) - 1 no digits: its value is rounding
        if beam[i] in (0.0, 1.1, 0.9):
            for key in ("thermal_fluxes", "fluxes"):
                np.testing.assert_allclose(got[key][:, i], want[key], rtol=1e-12)
        assert not np.isnan(got["thermal_fluxes"][:, i]).any()
