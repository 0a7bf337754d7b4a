"""The pooled differentiation passes take the sums of the general kernels: with the asteroid masses,
too, they keep unscaled series sums in their columns and fuse the scaling into the differences.

An ephemeris of two segments: epochs inside the first run the pooled passes, one epoch beyond
it the general ones.  The states at the common epochs: 1e-9 AU, and nearly all objects to the
bit (the sums that the two forms contract otherwise are one in hundreds)."""
import numpy as np
import pytest

from kete_b200 import synthetic
from kete_b200.synthetic import EPOCH

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("asteroids", [False, True])
def test_states_equal_the_general_passes(gpu, spk_path, tmp_path, asteroids):
    from kete_b200 import autodiff as A

    cut = 2457000.5 + 32.0 * 105  # EPOCH + 360
    paths = [str(tmp_path / "a.bsp"), str(tmp_path / "b.bsp")]
    synthetic.write_synthetic_spk(paths[0], jd_end=cut, asteroids=True)
    synthetic.write_synthetic_spk(paths[1], jd_start=cut, asteroids=True)
    inside = EPOCH + np.array([100.0, 300.0])
    beyond = np.append(inside, EPOCH + 370.0)
    gpu.spice.kernel_reload(paths)
    try:
        for n in (300, 1800):  # a warp an object, eight lanes
            pos, vel = synthetic.neo(n, seed=n)
            ng = np.repeat(synthetic.comet_nongrav(1e-8, 1e-9)[:, None], n, axis=1)
            ng[:, ::2] = 0.0
            jd0 = np.full(n, EPOCH)
            kw = dict(include_asteroids=asteroids, nongrav=ng)
            for run in (A.propagate_n_body_checkpointed, A.propagate_n_body_stm_arrays):
                a, b = (run(pos, vel, jd0, e, **kw)[0][:2] for e in (inside, beyond))
                assert np.isfinite(a).all() and np.abs(a - b).max() < 1e-9
                same = (a == b).all(axis=(0, 1)).mean()
                assert same > 0.95, (n, run.__name__, same)
    finally:
        gpu.spice.kernel_reload([spk_path])
