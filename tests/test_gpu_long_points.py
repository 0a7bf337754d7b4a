"""The system integration's forms: batches of up to 23 test particles with their points spread
over a block (two builds, each with and without the comet model), a thread per body above."""
import numpy as np
import pytest

from kete_b200 import synthetic
from kete_b200.synthetic import EPOCH

pytestmark = pytest.mark.gpu


def _states(n, seed):
    pos, vel = synthetic.main_belt(n, seed=seed)
    ng = np.stack([synthetic.comet_nongrav(1e-8, 1e-9)] * n, axis=1)
    ng[:, ::2] = 0.0
    return synthetic.ecl_to_eq(pos), synthetic.ecl_to_eq(vel), ng


@pytest.mark.parametrize("comets", [False, True])
@pytest.mark.parametrize("batch,n", [(1, 1), (1, 3), (12, 29), (13, 13), (14, 40), (23, 24), (24, 24)])
def test_block_edges_vs_oracle(gpu, oracle_spk, batch, n, comets):
    """1e-9 AU, the bound that the other system integrations are held to."""
    pos, vel, ng = _states(n, 3 + batch)
    ng = ng if comets else None
    p, v, pl, st = gpu.propagate_n_body_long_arrays(pos, vel, EPOCH, EPOCH + 120.0, None, ng, batch)
    op, ov, opl, ost = oracle_spk.propagate_n_body_vec(pos, vel, EPOCH, EPOCH + 120.0, ng=ng,
                                                       batch_size=batch)
    assert (st == 0).all() and (ost == 0).all()
    assert np.abs(p - op).max() < 1e-9 and np.abs(v - ov).max() < 1e-11
    assert np.abs(pl - opl).max() < 1e-9


def test_comets_beyond_a_wave_and_impact(gpu):
    """301 batches, more than one wave of blocks, and the first ten alone: bit for bit.  A particle inside the Sun ends its batch, and only that."""
    n, batch = 903, 3
    pos, vel, ng = _states(n, 8)
    first = [np.ascontiguousarray(x[:, :30]) for x in (pos, vel, ng)]
    run = lambda p, v, g: gpu.propagate_n_body_long_arrays(p, v, EPOCH, EPOCH - 40.0, None, g, batch)
    p, v, _, st = run(pos, vel, ng)
    q, w, _, st2 = run(*first)
    assert (st == 0).all() and (st2 == 0).all()
    assert np.array_equal(p[:, :30], q) and np.array_equal(v[:, :30], w)
    first[0][:, 4] = [1e-4, 0.0, 0.0]
    p2, _, _, st3 = run(*first)
    assert (st3[3:6] == 6).all() and (st3[:3] == 0).all() and (st3[6:] == 0).all()
    assert np.isnan(p2[:, 3:6]).all() and np.array_equal(p2[:, 6:], q[:, 6:])
