"""Every geometry of a block of several: large calls (8 and 16 geometries a block, up to four to
a warp) against the same inputs in slices of one geometry a warp, to the bit, and the oracle in
the middle of a block (1e-12 relative)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BANDS = {2: ([4700.0, 8000.0], False), 4: ([3352.6, 4602.8, 11098.4, 22640.5], True),
         8: ([9.0, 550.0, 2200.0, 3400.0, 4600.0, 12000.0, 22000.0, 1e5], False)}


@pytest.mark.parametrize("n", [9473, 18945])
@pytest.mark.parametrize("nb", BANDS)
def test_slots_of_a_block(gpu, oracle, n, nb):
    bands, cc = BANDS[nb]
    rng = np.random.default_rng(n + nb)
    r, th = rng.uniform(0.8, 40.0, n), rng.uniform(0, 2 * np.pi, n)
    s2obj = np.stack([r * np.cos(th), r * np.sin(th), rng.normal(0, 0.3, n)])
    th2 = rng.uniform(0, 2 * np.pi, n)
    s2obs = np.stack([np.cos(th2), np.sin(th2), np.zeros(n)])
    pv, h = rng.uniform(0.02, 0.6, n), rng.uniform(8, 20, n)
    diam = 1329.0 / np.sqrt(pv) * 10 ** (-h / 5)

    def run(sl):
        alb = np.repeat(pv[None, sl], nb, axis=0)
        args = (s2obj[:, sl], s2obs[:, sl], h[sl], 0.15, diam[sl], pv[sl])
        tail = (0.9, bands, alb, None, [100.0] * nb, cc)
        return (gpu.flux.neatm_arrays(*args, np.full(pv[sl].size, 1.1), *tail),
                gpu.flux.frm_arrays(*args, *tail))

    whole = run(slice(None))
    parts = [run(slice(a, a + 4000)) for a in range(0, n, 4000)]
    for m in range(2):
        for key, value in whole[m].items():
            sliced = np.concatenate([p[m][key] for p in parts], axis=-1)
            assert np.array_equal(value, sliced, equal_nan=True), (m, key)
    for i in (5, 6, 7, n // 2 + 3):
        want = oracle.neatm_total_flux(s2obj[:, i], s2obs[:, i], h[i], 0.15, diam[i], pv[i], 1.1, 0.9,
                                       bands, [pv[i]] * nb, None, [100.0] * nb, cc)
        np.testing.assert_allclose(whole[0]["fluxes"][:, i], want["fluxes"], rtol=1e-12)
