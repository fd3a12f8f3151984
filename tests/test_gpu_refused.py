"""Calls that a plan has no buffers for are refused: whole transforms (and test
hooks on the plan's q) on a shard of a plan, whose q buffers are the caller's,
and the phase entry points of a plan made without bound buffers."""
import ctypes

import numpy as np
import pytest

from wavemoth_b200 import _native
from wavemoth_b200 import lib as wlib

pytestmark = pytest.mark.gpu

ERR_ARG = 1


def _buffers(nside, lmax, nmaps):
    import torch
    alm = torch.zeros(((lmax + 1) * (lmax + 2) // 2, nmaps), dtype=torch.complex128, device="cuda")
    return alm, torch.zeros((12 * nside * nside, nmaps), dtype=torch.float64, device="cuda")


@pytest.mark.parametrize("part", [0, 1])
def test_whole_transforms_on_a_shard(part):
    import torch
    nside, lmax, nmaps = 8, 16, 2
    L = _native.lib()
    alm, f = _buffers(nside, lmax, nmaps)
    P = L.wavemoth_plan_shard(nside, lmax, lmax, nmaps, wlib.WAVEMOTH_DENSE, None, 2, part)
    assert P, wlib.last_error()
    work = np.zeros(2 * (lmax + 1) * 2 * nside * 2 * nmaps)
    calls = [lambda: L.wavemoth_execute_alm2map_device(P, alm.data_ptr(), f.data_ptr(), None),
             lambda: L.wavemoth_execute_map2alm_device(P, f.data_ptr(), alm.data_ptr(), None),
             lambda: L.wavemoth_alm2map_backward_device(P, f.data_ptr(), alm.data_ptr(), None),
             lambda: L.wavemoth_map2alm_iterative_device(P, f.data_ptr(), alm.data_ptr(), 1, None),
             lambda: L.wavemoth_legendre_alm2map_device(P, alm.data_ptr(), f.data_ptr(), None),
             lambda: L.wavemoth_legendre_map2alm_device(P, f.data_ptr(), alm.data_ptr(), None),
             lambda: L.wavemoth_get_work(P, work.ctypes.data_as(ctypes.POINTER(ctypes.c_double))),
             lambda: L.wavemoth_plan_set_hemisphere_mode(P, 1)]
    for call in calls:
        assert call() == ERR_ARG
        assert "shard" in wlib.last_error()
    torch.cuda.synchronize()
    L.wavemoth_destroy_plan(P)


def test_phases_of_a_plan_without_bound_buffers():
    import torch
    from wavemoth_b200.sht import Transform
    T = Transform(None, 8, 16, 2, dense=True)
    L = _native.lib()
    for call, which in ((L.wavemoth_perform_legendre_transforms, "input"), (L.wavemoth_perform_backward_ffts, "output")):
        call(T.plan_handle)
        assert L.wavemoth_plan_status(T.plan_handle) == ERR_ARG
        assert which in wlib.last_error()
    torch.cuda.synchronize()
    T.close()
