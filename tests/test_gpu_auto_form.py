"""The form the library picks by itself (MODE_AUTO with the default launch configuration): a warp
per object up to 4,096 objects, the warp-pooled form with its heavy objects in warps of their
own above.  Each against the general node kernel (variant 7) on the same inputs."""
import numpy as np
import pytest

from kete_b200 import synthetic
from kete_b200.synthetic import EPOCH

pytestmark = pytest.mark.gpu


def _inputs(n, seed):
    """A mix with comets (one delayed, one dust), a few long spans that the pooled form counts
    as heavy, targets outside the ephemeris, a NaN state, a NaN epoch and a zero span."""
    pos, vel, ng = synthetic.mixed(n, seed=seed, nongrav_frac=0.1)
    rng = np.random.default_rng(seed + 1)
    jd0 = np.full(n, EPOCH)
    jd1 = EPOCH + rng.uniform(-40.0, 40.0, n)
    jd1[::97] = EPOCH + 1200.0
    if n >= 30:
        jd1[3] = EPOCH + 1.0e5
        jd1[7] = EPOCH - 1.0e5
        pos[1, 11] = np.nan
        jd1[13] = np.nan
        jd1[17] = EPOCH
        ng[:, 19] = synthetic.comet_nongrav(1e-8, 1e-9)
        ng[9, 19] = 12.0
        ng[:, 23] = [2.0, 1e-3, 0, 0, 0, 0, 0, 0, 0, 0]
    return pos, vel, jd0, jd1, ng


@pytest.mark.parametrize("n", [1, 3, 33, 592, 4096, 4097, 9001])
def test_automatic_form_matches_general(gpu, n):
    from kete_b200 import tune

    pos, vel, jd0, jd1, ng = _inputs(n, seed=n)
    tune.set_config()
    p, v, st, det = gpu.propagate_n_body_arrays(pos, vel, jd0, jd1, nongrav=ng, with_details=True)
    p0, v0, st0, det0 = gpu.propagate_n_body_arrays(pos, vel, jd0, jd1, nongrav=ng, mode=2,
                                                    with_details=True)
    assert (st == st0).all()
    ok = st == 0
    assert ok.sum() >= n - 4 and np.isnan(p[:, ~ok]).all()
    # the same integration; both forms hold 1e-9 AU against the oracle
    assert np.abs(p[:, ok] - p0[:, ok]).max() < 1e-9
    assert np.abs(v[:, ok] - v0[:, ok]).max() < 1e-10
    assert np.abs(det["min_dist"][ok] - det0["min_dist"][ok]).max() < 1e-9
    assert (det["impact_id"] == det0["impact_id"]).all()


@pytest.mark.parametrize("n", [1, 250])
def test_automatic_form_oracle(gpu, oracle_spk, n):
    pos, vel, ng = synthetic.mixed(n, seed=5 + n)
    jd0 = np.full(n, EPOCH)
    jd1 = EPOCH + np.random.default_rng(n).uniform(-300.0, 300.0, n)
    p, v, st, det = gpu.propagate_n_body_arrays(pos, vel, jd0, jd1, nongrav=ng, with_details=True)
    op, _, ost, _, _ = oracle_spk.propagate_n_body(pos, vel, jd0, jd1, ng=ng)
    far = det["min_dist"] >= 0.01
    assert (st == ost).all() and (st == 0).all()
    assert np.abs(p - op)[:, far].max() < 1e-9


def test_automatic_form_asteroids_and_mixed_counts(gpu, spk_path, tmp_path):
    """The asteroids' plan (chained to the Sun), and series of different lengths."""
    counts = {10: 11, 1: 14, 2: 10, 3: 13, 399: 13, 301: 13, 4: 11, 5: 8, 6: 7, 7: 6, 8: 6}
    path = str(tmp_path / "mixed.bsp")
    synthetic.write_synthetic_spk(path, n_coef=counts, asteroids=True)
    gpu.spice.kernel_reload([path])
    try:
        for n in (50, 4500):
            pos, vel, jd0, jd1, ng = _inputs(n, seed=n + 2)
            for inc in (False, True):
                p, _, st = gpu.propagate_n_body_arrays(pos, vel, jd0, jd1, include_asteroids=inc,
                                                       nongrav=ng)
                p0, _, st0 = gpu.propagate_n_body_arrays(pos, vel, jd0, jd1, include_asteroids=inc,
                                                         nongrav=ng, mode=2)
                ok = st == 0
                assert (st == st0).all() and ok.sum() >= n - 4
                assert np.abs(p[:, ok] - p0[:, ok]).max() < 1e-9, (n, inc)
    finally:
        gpu.spice.kernel_reload([spk_path])
