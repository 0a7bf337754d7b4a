"""The thermal kernel at the edges of its blocks (4, 8 or 16 geometries a block by the count),
with one to eight bands, and with facets too cold for their bands (the plain form), against the
oracle: fluxes 1e-12 relative, magnitudes 1e-9."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BANDS = {1: [12000.0], 2: [4700.0, 8000.0], 3: [5.0, 4602.8, 22088.3],
         4: [3352.6, 4602.8, 11098.4, 22640.5], 5: [550.0, 1200.0, 4700.0, 8000.0, 1e6],
         8: [9.0, 550.0, 2200.0, 3400.0, 4600.0, 12000.0, 22000.0, 1e5]}


def _inputs(n, nb, seed):
    rng = np.random.default_rng(seed)
    r, th = rng.uniform(0.8, 40.0, n), rng.uniform(0, 2 * np.pi, n)
    s2obj = np.stack([r * np.cos(th), r * np.sin(th), rng.normal(0, 0.3, n)])
    th2 = rng.uniform(0, 2 * np.pi, n)
    s2obs = np.stack([np.cos(th2), np.sin(th2), np.zeros(n)])
    pv = rng.uniform(0.02, 0.6, n)
    h = rng.uniform(8, 20, n)
    diam = 1329.0 / np.sqrt(pv) * 10 ** (-h / 5)
    return s2obj, s2obs, h, pv, diam, np.repeat(pv[None], nb, axis=0)


@pytest.mark.parametrize("n", [1, 5, 9471, 9473, 18945])
@pytest.mark.parametrize("nb,cc", [(1, False), (2, False), (3, False), (4, True), (5, False),
                                   (8, False)])
def test_thermal_blocks(gpu, oracle, n, nb, cc):
    s2obj, s2obs, h, pv, diam, alb = _inputs(n, nb, n + nb)
    bands = BANDS[nb]
    beam = np.full(n, 1.1)
    neatm = gpu.flux.neatm_arrays(s2obj, s2obs, h, 0.15, diam, pv, beam, 0.9, bands, alb, None,
                                  [100.0] * nb, cc)
    frm = gpu.flux.frm_arrays(s2obj, s2obs, h, 0.15, diam, pv, 0.9, bands, alb, None, [100.0] * nb,
                              cc)
    for i in sorted({0, n // 2, n - 2, n - 1} & set(range(n))):
        on = oracle.neatm_total_flux(s2obj[:, i], s2obs[:, i], h[i], 0.15, diam[i], pv[i], 1.1, 0.9,
                                     bands, [pv[i]] * nb, None, [100.0] * nb, cc)
        of = oracle.frm_total_flux(s2obj[:, i], s2obs[:, i], h[i], 0.15, diam[i], pv[i], 0.9, bands,
                                   [pv[i]] * nb, None, [100.0] * nb, cc)
        for got, want in ((neatm, on), (frm, of)):
            np.testing.assert_allclose(got["thermal_fluxes"][:, i], want["thermal_fluxes"], rtol=1e-12)
            np.testing.assert_allclose(got["fluxes"][:, i], want["fluxes"], rtol=1e-12)
            np.testing.assert_allclose(got["magnitudes"][:, i], want["magnitudes"], atol=1e-9)
            np.testing.assert_allclose(got["v_band_magnitude"][i], want["v_band_magnitude"], atol=1e-9)
