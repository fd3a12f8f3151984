"""Which kernels a split-precision plan runs, and both of its routes.

Plans of few maps on images of at least 2^22 Legendre elements run on the FP64
units; a plan with a wait limit set keeps the split GEMMs (whose waits the
limit bounds), which is how these tests reach them at every size.  Bounds:
the FP64 route is the FP64 plan's kernels on equal tables, so equal bits; the
split GEMMs keep 42 bits of each operand relative to its largest entry, 1e-10
of the largest output here.
"""
import numpy as np
import pytest

from oracle import sht as osht
from wavemoth_b200 import _native

from .plans import plan_file

pytestmark = pytest.mark.gpu


def _plan(path, nside, lmax, nmaps, precision, gemms=False):
    from wavemoth_b200.sht import Transform
    T = Transform(path, nside, lmax, nmaps, precision=precision, dense=path is None)
    if gemms:
        assert _native.lib().wavemoth_plan_set_wait_limit(T.plan_handle, 1 << 26) == 0
    return T


def _both_ways(T, alm, nside, lmax):
    import torch
    f = T.alm2map(alm, out=torch.full((T.npix, T.nmaps), float("nan"), dtype=torch.float64, device="cuda"))
    a = T.map2alm(f, out=torch.full((T.nalm, T.nmaps), float("nan"), dtype=torch.complex128, device="cuda"))
    torch.cuda.synchronize()
    T.device_status()
    return f, a


def _close(got, want):
    return float((got - want).abs().max()) <= 1e-10 * float(want.abs().max())


@pytest.mark.parametrize("nmaps", [1, 3, 10])
def test_few_maps_on_a_large_plan_equal_the_fp64_plan(nmaps):
    torch = pytest.importorskip("torch")
    nside, lmax = 128, 300
    alm = torch.from_numpy(osht.random_alm(lmax, nmaps, seed=nmaps)).cuda()
    S, D = (_plan(None, nside, lmax, nmaps, p) for p in ("split", "double"))
    got, want = _both_ways(S, alm, nside, lmax), _both_ways(D, alm, nside, lmax)
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
    # and the GEMMs on the same plan, then the FP64 route again (q and X rows
    # of one route must not show in the other)
    L = _native.lib()
    assert L.wavemoth_plan_set_wait_limit(S.plan_handle, 1 << 26) == 0
    gemms = _both_ways(S, alm, nside, lmax)
    assert not torch.equal(gemms[0], want[0])
    assert _close(gemms[0], want[0]) and _close(gemms[1], want[1])
    assert L.wavemoth_plan_set_wait_limit(S.plan_handle, 0) == 0
    again = _both_ways(S, alm, nside, lmax)
    assert torch.equal(again[0], want[0]) and torch.equal(again[1], want[1])
    S.close()
    D.close()


@pytest.mark.parametrize("nside,lmax,nmaps", [(16, 33, 2), (32, 95, 40), (64, 259, 3), (65, 287, 33), (128, 255, 12)])
@pytest.mark.parametrize("precision", ["split", "split-generate"])
def test_gemms_with_ragged_tiles(nside, lmax, nmaps, precision):
    """Row and column counts just above multiples of 16 and 128: last tiles of
    one 16-row block, K chunks that end before a tile's first column starts."""
    torch = pytest.importorskip("torch")
    alm = torch.from_numpy(osht.random_alm(lmax, nmaps, seed=lmax)).cuda()
    S, D = _plan(None, nside, lmax, nmaps, precision, gemms=True), _plan(None, nside, lmax, nmaps, "double")
    got, want = _both_ways(S, alm, nside, lmax), _both_ways(D, alm, nside, lmax)
    assert _close(got[0], want[0]) and _close(got[1], want[1])
    S.close()
    D.close()


@pytest.mark.parametrize("nside,lmax,chunk,nmaps", [(64, 150, 16, 5), (128, 256, 64, 33)])
def test_gemms_of_interpolation_levels(nside, lmax, chunk, nmaps):
    torch = pytest.importorskip("torch")
    path = plan_file(nside, lmax, chunk, 1e-12, 1e-10, workers=4, max_levels=1)
    alm = torch.from_numpy(osht.random_alm(lmax, nmaps, seed=3)).cuda()
    S = _plan(path, nside, lmax, nmaps, "split", gemms=True)
    G = _plan(path, nside, lmax, nmaps, "split-generate", gemms=True)
    D = _plan(path, nside, lmax, nmaps, "double")
    got, gen, want = (_both_ways(T, alm, nside, lmax) for T in (S, G, D))
    assert torch.equal(got[0], gen[0]) and torch.equal(got[1], gen[1])
    assert _close(got[0], want[0]) and _close(got[1], want[1])
    for T in (S, G, D):
        T.close()
