"""The warp-per-object form and the pooled variants 9 and 10 are one integration: the same states,
counters and closest approaches to the bit, whatever form an object gets by the count of its
call.  The same for the differentiation passes, a warp per object or eight lanes."""
import numpy as np
import pytest

from kete_b200 import synthetic
from kete_b200.synthetic import EPOCH

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("asteroids", [False, True])
def test_propagation_forms_are_equal(gpu, spk_path, tmp_path, asteroids):
    from kete_b200 import tune

    path = str(tmp_path / "asteroids.bsp")
    synthetic.write_synthetic_spk(path, asteroids=True)
    gpu.spice.kernel_reload([path])
    n = 1500
    pos, vel, ng = synthetic.mixed(n, seed=9, neo_frac=0.3, nongrav_frac=0.2)
    ng[:, 5] = synthetic.comet_nongrav(1e-8, 1e-9)
    ng[9, 5] = 12.0
    ng[:, 6] = [2.0, 1e-3, 0, 0, 0, 0, 0, 0, 0, 0]
    jd0 = np.full(n, EPOCH)
    jd1 = EPOCH + np.random.default_rng(1).uniform(-400.0, 400.0, n)
    kw = dict(include_asteroids=asteroids, nongrav=ng, with_details=True)
    try:
        tune.set_config()
        want = gpu.propagate_n_body_arrays(pos, vel, jd0, jd1, **kw)
        for variant in (9, 10):
            for refill in (0, 1):
                tune.set_config(variant=variant, refill=refill)
                got = gpu.propagate_n_body_arrays(pos, vel, jd0, jd1, **kw)
                for a, b in zip(want[:3], got[:3]):
                    assert np.array_equal(a, b), (variant, refill)
                for key in want[3]:
                    assert np.array_equal(want[3][key], got[3][key]), (variant, refill, key)
    finally:
        tune.set_config()
        gpu.spice.kernel_reload([spk_path])


@pytest.mark.parametrize("asteroids", [False, True])
def test_forward_pass_forms_are_equal(gpu, spk_path, tmp_path, asteroids):
    """1776 objects take a warp each, 1777 eight lanes."""
    from kete_b200 import autodiff as A

    path = str(tmp_path / "asteroids.bsp")
    synthetic.write_synthetic_spk(path, asteroids=True)
    gpu.spice.kernel_reload([path])
    n = 1777
    pos, vel, ng = synthetic.mixed(n, seed=10, neo_frac=0.3, nongrav_frac=0.5)
    jd0 = np.full(n, EPOCH)
    epochs = EPOCH + np.array([30.0, 400.0])
    try:
        out = []
        for k in (n, n - 1):
            s, st, ck = A.propagate_n_body_checkpointed(
                *(np.ascontiguousarray(x[..., :k]) for x in (pos, vel, jd0)), epochs,
                include_asteroids=asteroids, nongrav=np.ascontiguousarray(ng[:, :k]))
            assert (st == 0).all()
            out.append((s, ck.count, ck.ckpt, ck.capacity))
        (s1, c1, k1, cap), (s4, c4, k4, cap4) = out
        assert np.array_equal(s1[..., :n - 1], s4) and np.array_equal(c1[:n - 1], c4)
        assert cap == cap4
        for i in range(0, n - 1, 7):
            assert np.array_equal(k1[i, :c1[i], :35], k4[i, :c4[i], :35])
    finally:
        gpu.spice.kernel_reload([spk_path])
