"""Closest approach of the warp-pooled forms against the general node kernel (mode 2),
which takes the bodies in the plan's order.  Distances to 1e-9 AU, the bound of the states."""
import numpy as np
import pytest

from kete_b200 import synthetic
from kete_b200.synthetic import EPOCH

pytestmark = pytest.mark.gpu


@pytest.fixture
def asteroid_spk(gpu, spk_path, tmp_path):
    path = str(tmp_path / "asteroids.bsp")
    synthetic.write_synthetic_spk(path, asteroids=True)
    gpu.spice.kernel_reload([path])
    yield gpu
    gpu.spice.kernel_reload([spk_path])


def _compare(gpu, pos, vel, jd0, jd1, config=None, **kw):
    from kete_b200 import tune

    kw["with_details"] = True
    p0, _, st0, d0 = gpu.propagate_n_body_arrays(pos, vel, jd0, jd1, mode=2, **kw)
    try:
        if config:
            tune.set_config(**config)
        p, _, st, d = gpu.propagate_n_body_arrays(pos, vel, jd0, jd1, **kw)
    finally:
        tune.set_config()
    assert (st == st0).all()
    assert np.array_equal(np.isnan(p), np.isnan(p0))
    assert np.array_equal(d["impact_id"], d0["impact_id"])
    assert np.abs(d["impact_jd"] - d0["impact_jd"]).max() < 1e-9
    assert np.abs(d["min_dist"] - d0["min_dist"]).max() < 1e-9
    return st0, d0


@pytest.mark.parametrize("n,config", [
    (1, None), (64, None), (4500, None), (130, dict(variant=9, refill=0)),
    (130, dict(variant=9, refill=1)), (131, dict(variant=10, refill=0)),
    (131, dict(variant=10, refill=1))])
def test_min_dist_with_the_asteroids(asteroid_spk, n, config):
    """The bodies without velocity are 13: the last one has no partner in the pairs.  Near-Earth
    objects pass the barycentre closer than any planet."""
    pos, vel = synthetic.neo(n, seed=n)
    rng = np.random.default_rng(n)
    jd0 = np.full(n, EPOCH)
    jd1 = EPOCH + rng.uniform(-60.0, 60.0, n)
    jd1[::5] = EPOCH  # zero spans: the state's own distances
    pos[:, 0] = [0.25, 0.05, 0.02]
    st, d = _compare(asteroid_spk, pos, vel, jd0, jd1, config, include_asteroids=True)
    assert (st == 0).all() and d["min_dist"][0] > 0.0
