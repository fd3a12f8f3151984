"""Plan files whose depth-1 roots are too large for the FP64 level kernels
(leaves of half the rings and more): FP64 plans run them on the generic
kernels, split plans of few maps on the split GEMMs.  Checked against a dense
plan, which has no interpolation, and the split plan against its own GEMMs, bit
for bit.  Bound: an interpolative decomposition of precision eps = 1e-12 of k
out of n columns errs by up to sqrt(1 + k (n - k)) eps, 8e-10 for k = 200 and
n = 3072; 1e-9 with the split GEMMs' 1e-10."""
import os

import pytest

from oracle import sht as osht
from wavemoth_b200 import _native

from .plans import plan_file

pytestmark = pytest.mark.gpu


def _run(T, alm, f):
    import torch
    out = T.alm2map(alm), T.map2alm(f)
    torch.cuda.synchronize()
    T.device_status()
    return out


def _close(got, want):
    return all(float((g - w).norm()) <= 1e-9 * float(w.norm()) for g, w in zip(got, want))


def _compare(nside, lmax, nmaps, precision, gemms):
    import torch
    from wavemoth_b200.sht import Transform
    path = plan_file(nside, lmax, nside, 1e-12, 1e-10, workers=min(8, os.cpu_count()), max_levels=1)
    alm = torch.from_numpy(osht.random_alm(lmax, nmaps, seed=nside)).cuda()
    D = Transform(None, nside, lmax, nmaps, dense=True)
    f = D.alm2map(alm)
    want = _run(D, alm, f)
    D.close()
    T = Transform(path, nside, lmax, nmaps, precision=precision)
    got = _run(T, alm, f)
    if gemms:
        assert _native.lib().wavemoth_plan_set_wait_limit(T.plan_handle, 1 << 26) == 0
        again = _run(T, alm, f)
        assert torch.equal(got[0], again[0]) and torch.equal(got[1], again[1])
    T.close()
    assert _close(got, want)


@pytest.mark.parametrize("nmaps", [1, 5])
def test_fp64_plan(nmaps):
    _compare(2048, 24, nmaps, "double", False)


def test_split_plan_of_few_maps():
    """2^22 Legendre elements and more, where plans of few maps run in FP64 if
    the level kernels take their roots."""
    assert _native.lib().wm_host_level_fits(3072, 200) == 0
    _compare(1536, 400, 3, "split", True)
