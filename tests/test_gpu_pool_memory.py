"""Device memory of a loaded ephemeris: the records once in the general layout and once in the
pooled kernels', the planets' series shared by the plans with and without the asteroids."""
import numpy as np
import pytest

from kete_b200 import synthetic

pytestmark = pytest.mark.gpu


def test_records_are_held_twice_at_most(gpu, spk_path, tmp_path):
    import torch

    path = str(tmp_path / "fine.bsp")
    # records of a quarter day: 14 MB in the general layout
    synthetic.write_synthetic_spk(path, jd_start=2459700.5, jd_end=2460300.5, record_days=0.25,
                                  moon_record_days=0.25, asteroids=True)
    general = 16 * 2400 * (4 + 3 * 14) * 8
    gpu.spice.kernel_reload([spk_path])
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    try:
        gpu.spice.kernel_reload([path])
        held = before - torch.cuda.mem_get_info()[0]
        pos, vel = synthetic.main_belt(3, seed=1)
        for asteroids in (False, True):
            _, _, st = gpu.propagate_n_body_arrays(pos, vel, np.full(3, synthetic.EPOCH),
                                                   np.full(3, synthetic.EPOCH + 30.0),
                                                   include_asteroids=asteroids)
            assert (st == 0).all()
    finally:
        gpu.spice.kernel_reload([spk_path])
    assert general < held < 2.2 * general
