"""An installed launch configuration is what the automatic mode runs, the library's own start
values included; without arguments set_config goes back to the automatic choice."""
import numpy as np
import pytest

from kete_b200 import synthetic
from kete_b200.synthetic import EPOCH

pytestmark = pytest.mark.gpu


def _launches(gpu, n=100):
    import ctypes

    from kete_b200 import _lib

    f = _lib.lib().kete_b200_kernel_launches
    f.restype = ctypes.c_int64
    pos, vel = synthetic.main_belt(n, seed=1)
    before = f()
    _, _, st = gpu.propagate_n_body_arrays(pos, vel, np.full(n, EPOCH), np.full(n, EPOCH + 5.0))
    assert (st == 0).all()
    return f() - before


def test_installed_start_values_are_run(gpu):
    from kete_b200 import _lib, tune

    tune.set_config()
    automatic = _launches(gpu)
    try:
        tune.set_config(variant=7, refill=0)
        installed = _launches(gpu)
        tune.set_config(variant=6, refill=0)  # the same launches with another register cap
        assert installed == _launches(gpu) == 4 and automatic == 2
        tune.set_config()
        assert _launches(gpu) == automatic
        L = _lib.lib()
        _lib.check(L.kete_b200_set_launch_config(7, 0, 128))
        assert _launches(gpu) == 4
        assert L.kete_b200_set_launch_config(-1, 0, 128) != 0  # refused as ever
        assert L.kete_b200_set_launch_config(11, 0, 128) != 0
    finally:
        tune.set_config()
    assert _launches(gpu) == automatic
    assert tune.current()["variant"] == 7 and tune.current()["refill"] == 0
    cur = tune.current()  # round trips, from both states
    tune.set_config(variant=7, refill=0)
    inst = tune.current()
    try:
        tune.set_config(**cur)
        assert _launches(gpu) == automatic
        tune.set_config(**inst)
        assert _launches(gpu) == 4
    finally:
        tune.set_config()


def test_allocation_free_call_runs_what_is_installed(gpu):
    import ctypes

    import torch

    from kete_b200 import _lib, tune

    L = _lib.lib()
    L.kete_b200_kernel_launches.restype = ctypes.c_int64
    n = 100
    pos, vel = synthetic.main_belt(n, seed=1)
    dev = [torch.as_tensor(np.ascontiguousarray(x), device="cuda") for x in
           (pos, vel, np.full(n, EPOCH), np.full(n, EPOCH + 5.0))]
    out = [torch.empty((3, n), dtype=torch.float64, device="cuda") for _ in range(2)]
    st = torch.empty(n, dtype=torch.int32, device="cuda")
    p = ctypes.c_void_p
    f = L.kete_b200_propagate_n_body_noalloc
    f.argtypes = [ctypes.c_int64, p, p, p, p, ctypes.c_int, ctypes.c_int64, ctypes.c_int] + [p] * 9

    def launches():
        before = L.kete_b200_kernel_launches()
        _lib.check(f(n, *(x.data_ptr() for x in dev), 2, 10, 0, None, out[0].data_ptr(),
                     out[1].data_ptr(), st.data_ptr(), None, None, None, None,
                     torch.cuda.current_stream().cuda_stream))
        torch.cuda.synchronize()
        assert bool((st == 0).all())
        return L.kete_b200_kernel_launches() - before

    tune.set_config()
    try:
        assert launches() == 2
        tune.set_config(variant=7, refill=0)
        assert launches() == 4
    finally:
        tune.set_config()
