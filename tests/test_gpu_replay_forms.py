"""Replays of checkpoint blocks are the forward pass's own steps: the gradients of the two
adjoint forms are equal to the bit, and match the transposed sensitivities, where a block ends
and the next begins inside a segment (spans of hundreds of days), with the asteroid masses, with
an ephemeris of two segments and with more records than one pass of the sweep takes.

Against the sensitivities: the states of the two passes agree to 1e-9 AU (the bound of every
form); over two years that moves a sensitivity by up to some 100 times as much relative to
itself, so 1e-6 of each parameter group, for objects that keep 0.05 AU from the planets (closer
approaches amplify further).  A block that ends at another step is off by days: 1e-3 and more."""
import numpy as np
import pytest

from kete_b200 import synthetic
from kete_b200.synthetic import EPOCH

pytestmark = pytest.mark.gpu


def _inputs(n, seed):
    pos, vel = synthetic.neo(n, seed=seed)
    rng = np.random.default_rng(seed)
    ng = np.stack([synthetic.comet_nongrav(*rng.normal(0.0, 1.0, 2) * (2e-8, 2e-9))
                   for _ in range(n)], axis=1)
    ng[:, ::3] = 0.0
    return pos, vel, np.full(n, EPOCH), ng


def _gradients(A, ck, seed):
    out = []
    try:
        for form in (0, 1):
            A.set_adjoint_form(form)
            g, st = A.propagate_n_body_adjoint(ck, seed)
            assert (st == 0).all()
            out.append(g)
    finally:
        A.set_adjoint_form(0)
    return out


def _check(gpu, n, epochs, asteroids, **kw):
    from kete_b200 import autodiff as A

    pos, vel, jd0, ng = _inputs(n, n)
    args = dict(include_asteroids=asteroids, nongrav=ng)
    _, st, ck = A.propagate_n_body_checkpointed(pos, vel, jd0, epochs, **kw, **args)
    assert (st == 0).all()
    seed = np.random.default_rng(2).normal(size=(len(epochs), 6, n))
    g0, g1 = _gradients(A, ck, seed)
    assert np.array_equal(g0, g1)
    _, m, st = A.propagate_n_body_stm_arrays(pos, vel, jd0, epochs, **args)
    far = st == 0
    for e in epochs:
        far &= gpu.propagate_n_body_arrays(pos, vel, jd0, np.full(n, e), mode=2, with_details=True,
                                           **args)[3]["min_dist"] > 0.05
    assert far.sum() > 0.7 * n
    ref = np.einsum("kcn,kcpn->pn", seed, m.reshape(len(epochs), 6, 8, n))
    for rows in (slice(0, 3), slice(3, 6)):
        scale = np.abs(ref[rows]).max(axis=0)
        err = np.abs(g0[rows] - ref[rows]).max(axis=0) / scale
        assert err[far].max() <= 1e-6


# 400 objects: a warp an object in the forward pass; 1900: eight lanes
@pytest.mark.parametrize("n", [400, 1900])
@pytest.mark.parametrize("asteroids", [False, True])
@pytest.mark.parametrize("segments", [1, 2])
def test_gradients_across_blocks(gpu, spk_path, tmp_path, n, asteroids, segments):
    """Two epochs over two years.  Two segments: the fast plan's window ends between the epochs,
    so that the first epoch's blocks lie inside it and the second's outside."""
    paths = [str(tmp_path / f"{k}.bsp") for k in range(segments)]
    cut = 2457000.5 + 32.0 * 105  # EPOCH + 360
    if segments == 1:
        synthetic.write_synthetic_spk(paths[0], asteroids=True)
    else:
        synthetic.write_synthetic_spk(paths[0], jd_end=cut, asteroids=True)
        synthetic.write_synthetic_spk(paths[1], jd_start=cut, asteroids=True)
    gpu.spice.kernel_reload(paths)
    try:
        _check(gpu, n, EPOCH + np.array([340.0, 730.0]), asteroids)
    finally:
        gpu.spice.kernel_reload([spk_path])


def test_records_beyond_one_pass(gpu, spk_path, tmp_path):
    """60,000 objects of up to 36 blocks (17 GiB of records) pass by pass, against the other form
    and, for the first 500, against a call of their own."""
    import torch

    from kete_b200 import autodiff as A

    path = str(tmp_path / "asteroids.bsp")
    synthetic.write_synthetic_spk(path, asteroids=True)
    gpu.spice.kernel_reload([path])
    try:
        n, few = 60_000, 500
        dev = [torch.as_tensor(x, device="cuda") for x in _inputs(n, 5)]
        epochs = torch.as_tensor(EPOCH + np.linspace(10.0, 300.0, 30), device="cuda")
        seed = torch.as_tensor(np.random.default_rng(4).normal(size=(30, 6, n)), device="cuda")

        def run(k):
            pos, vel, jd0, ng = (x[..., :k].contiguous() for x in dev)
            _, st, ck = A.propagate_n_body_checkpointed(pos, vel, jd0, epochs, capacity=60, nongrav=ng,
                                                        include_asteroids=True)
            assert bool((st == 0).all())
            assert k == few or n * ck.capacity * 17 * 36 * 8 > 8 << 30
            return _gradients(A, ck, seed[..., :k].contiguous()), ck.count

        (g0, g1), count = run(n)
        assert int(count.max()) > 30
        assert torch.equal(g0, g1)
        (h0, h1), _ = run(few)
        assert torch.equal(g0[:, :few], h0) and torch.equal(h0, h1)
    finally:
        gpu.spice.kernel_reload([spk_path])


def test_foreign_checkpoint_is_reported(gpu):
    """A block that does not end where the next one begins gives a status and NaN."""
    from kete_b200 import autodiff as A

    n = 20
    pos, vel, jd0, ng = _inputs(n, 77)
    epochs = EPOCH + np.array([700.0])
    _, st, ck = A.propagate_n_body_checkpointed(pos, vel, jd0, epochs, nongrav=ng)
    assert (st == 0).all() and ck.count[3] > 2
    ck.ckpt[3, 1, 0] += 0.5  # the second block of one object starts half a day later
    seed = np.random.default_rng(2).normal(size=(1, 6, n))
    for form in (0, 1):
        A.set_adjoint_form(form)
        try:
            g, gst = A.propagate_n_body_adjoint(ck, seed)
        finally:
            A.set_adjoint_form(0)
        assert gst[3] != 0 and np.isnan(g[:, 3]).all()
        assert (np.delete(gst, 3) == 0).all() and np.isfinite(np.delete(g, 3, axis=1)).all()
