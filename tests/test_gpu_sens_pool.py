"""The differentiation passes on pooled ephemeris records, at the sizes where their forms change
(a warp per object or eight lanes, two block counts of the sensitivities) and with objects that
they leave to the general kernels: started outside the ephemeris, a NaN state, a comet
with a delay.  States and sensitivities against the one-object-per-thread form, with the
bounds that it is held to elsewhere (1e-9 AU, 1e-7 of a column); the gradients against the
transposed sensitivities (1e-8 of a parameter group); the replays bit for bit where both
read positions from the cache."""
import numpy as np
import pytest

from kete_b200 import synthetic
from kete_b200.synthetic import EPOCH

pytestmark = pytest.mark.gpu

EPOCHS = EPOCH + np.array([12.5, 12.5, 47.0, -31.0])


def _inputs(n):
    pos, vel = synthetic.main_belt(n, seed=n)
    rng = np.random.default_rng(n + 1)
    ng = np.stack([synthetic.comet_nongrav(*rng.normal(0.0, 1.0, 2) * (2e-8, 2e-9))
                   for _ in range(n)], axis=1)
    ng[:, ::3] = 0.0
    jd0 = EPOCH + rng.uniform(-5.0, 5.0, n)
    bad = []
    if n > 20:
        ng[:, 5] = [2.0, 1e-3, 0, 0, 0, 0, 0, 0, 0, 0]
        jd0[7], jd0[11] = EPOCH + 1.0e5, EPOCH - 1.0e5
        pos[1, 13] = np.nan
        ng[:, 17] = synthetic.comet_nongrav(1e-8, 1e-9)
        ng[9, 17] = 12.0
        bad = [7, 11, 13, 17]
    return pos, vel, jd0, ng, bad


@pytest.mark.parametrize("n,asteroids", [(1, False), (3, True), (133, True), (1184, False),
                                         (1185, False), (1776, False), (1777, True)])
def test_pooled_passes_match_general(gpu, spk_path, tmp_path, n, asteroids):
    from kete_b200 import autodiff as A

    if asteroids:
        path = str(tmp_path / "asteroids.bsp")
        synthetic.write_synthetic_spk(path, asteroids=True)
        gpu.spice.kernel_reload([path])
    try:
        _check(A, n, asteroids)
    finally:
        if asteroids:
            gpu.spice.kernel_reload([spk_path])


def _check(A, n, asteroids):

    pos, vel, jd0, ng, bad = _inputs(n)
    kw = dict(include_asteroids=asteroids, nongrav=ng)
    K = len(EPOCHS)
    states, st, ck = A.propagate_n_body_checkpointed(pos, vel, jd0, EPOCHS, capacity=8, **kw)
    s1, m1, st1 = A.propagate_n_body_stm_arrays(pos, vel, jd0, EPOCHS, **kw)
    seed = np.random.default_rng(2).normal(size=(K, 6, n))
    try:
        A.set_sensitivity_form(1)
        s0, m0, st0 = A.propagate_n_body_stm_arrays(pos, vel, jd0, EPOCHS, **kw)
        g = []
        for form in (0, 1):
            A.set_adjoint_form(form)
            g.append(A.propagate_n_body_adjoint(ck, seed)[0])
    finally:
        A.set_sensitivity_form(0)
        A.set_adjoint_form(0)
    ok = np.ones(n, bool)
    ok[bad] = False
    assert (st0[ok] == 0).all() and (st0[~ok] != 0).all()
    assert (st == st0).all() and (st1 == st0).all()
    for s in (states, s1):
        assert np.abs(s - s0)[:, :, ok].max() < 1e-9
        assert np.array_equal(np.isnan(s), np.isnan(s0))
    err = (np.abs(m1 - m0).max(axis=1) / np.abs(m0).max(axis=1))[..., ok]
    assert np.nanmax(err) < 1e-7
    assert np.array_equal(np.isnan(m1), np.isnan(m0))
    if not asteroids:  # the general replay takes them without the cache of rounded positions
        assert np.array_equal(g[0], g[1], equal_nan=True)
    ref = np.einsum("kcn,kcpn->pn", seed, m1.reshape(K, 6, 8, n))[:, ok]
    for rows in (slice(0, 3), slice(3, 6)):
        scale = np.abs(ref[rows]).max(axis=0)
        for grad in g:
            assert (np.abs(grad[rows][:, ok] - ref[rows]).max(axis=0) <= 1e-8 * scale).all()
    assert np.isnan(g[0][:, ~ok]).all()
