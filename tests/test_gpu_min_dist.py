"""Closest approach and impact of the warp-pooled forms against the general node kernel (mode 2),
which takes the bodies in the plan's order.  Distances to 1e-9 AU, the bound of the states."""
import numpy as np
import pytest

from kete_b200 import synthetic
from kete_b200.synthetic import EPOCH

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def asteroid_path(tmp_path_factory):
    path = str(tmp_path_factory.mktemp("spk") / "asteroids.bsp")
    return synthetic.write_synthetic_spk(path, asteroids=True)


@pytest.fixture
def asteroid_spk(gpu, spk_path, asteroid_path):
    gpu.spice.kernel_reload([asteroid_path])
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


RADIUS = {1: 1.63139354095098e-05, 2: 4.04537843465442e-05, 399: 4.33036684926559e-05,
          4: 2.27021279387769e-05}


def _colliding(gpu, n, body):
    """Objects of which the first starts inside the body and the second a step outside it."""
    pos, vel = synthetic.main_belt(n, seed=3)
    state = gpu.spice.get_states_arrays(body, [EPOCH], center=10)[0][:, 0]
    for k, (r, v) in enumerate(((0.7 * RADIUS[body], 0.0), (RADIUS[body] + 1e-6, -0.002))):
        u = np.array([0.6, -0.64, 0.48])
        pos[:, k] = state[:3] + r * u
        vel[:, k] = state[3:] + v * u
    jd0 = np.full(n, EPOCH)
    jd1 = EPOCH + np.random.default_rng(n).uniform(1.0, 30.0, n)
    jd1[1] = EPOCH + 0.004  # one step
    return pos, vel, jd0, jd1


@pytest.mark.parametrize("n,config", [(2, None), (4500, None), (70, dict(variant=9, refill=1)),
                                      (70, dict(variant=10, refill=0))])
@pytest.mark.parametrize("body", RADIUS)
@pytest.mark.parametrize("asteroids", [False, True])
def test_impacts_do_not_depend_on_the_form(asteroid_spk, n, config, body, asteroids):
    """The bodies after the struck one in the plan do not count for the closest approach."""
    st, d = _compare(asteroid_spk, *_colliding(asteroid_spk, n, body), config,
                     include_asteroids=asteroids)
    assert (st[:2] == 6).all() and (d["impact_id"][:2] == body).all()


@pytest.mark.parametrize("other", [2, 399, 4])
def test_impact_inside_two_bodies(gpu, spk_path, tmp_path, other):
    """Inside two bodies at once (a second body on Mercury's path) the first of the plan counts."""
    path = str(tmp_path / "twice.bsp")
    segs = synthetic.read_daf_segments(spk_path)
    mercury = next(s for s in segs if s[0] == 1)
    synthetic.write_daf_spk(path, [(other, *mercury[1:]) if s[0] == other else s for s in segs])
    gpu.spice.kernel_reload([path])
    try:
        state = gpu.spice.get_states_arrays(1, [EPOCH], center=10)[0][:, 0]
        pos = (state[:3] + [0.0, 1e-5, 0.0])[:, None].copy()
        vel = state[3:][:, None].copy()
        st, d = _compare(gpu, pos, vel, np.array([EPOCH]), np.array([EPOCH + 5.0]))
        assert st[0] == 6 and d["impact_id"][0] == 1
    finally:
        gpu.spice.kernel_reload([spk_path])
