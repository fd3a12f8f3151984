"""FP64 residual products (legendre_direct.cu) at the edges of their tiles:
matrices of a few rows (all dense), row counts around multiples of the
map2alm tile (8 segments of 4 to 16 rows) and of the alm2map chunk (128
rows), column counts around multiples of 4, 32, 128 and 256, and every
number-of-vectors variant, against the oracle's dense FP64 transform.

Tolerance: a column's recurrence makes at most lmax / 2 steps of two
roundings each, coherent over the sum in the worst case, so lmax 2^-52; the
transform's own sums and FFTs stay far below that.  Factor 4 for the oracle,
whose recurrence rounds as well.
"""
import ctypes

import numpy as np
import pytest

from oracle import sht as osht

from .plans import plan_file, rel

pytestmark = pytest.mark.gpu

SIZES = [(1, 2), (2, 1), (4, 9), (5, 14), (16, 31), (16, 33), (33, 65), (64, 191), (65, 130), (128, 255), (130, 259)]


def _tol(lmax):
    return 4 * max(lmax, 16) * 2.0 ** -52


def _transform(nside, lmax, nmaps):
    from wavemoth_b200.sht import Transform
    return Transform(None, nside, lmax, nmaps, dense=True)


@pytest.mark.parametrize("nside,lmax", SIZES)
def test_against_dense_oracle(nside, lmax):
    torch = pytest.importorskip("torch")
    nmaps = 3
    alm = osht.random_alm(lmax, nmaps, seed=nside + lmax)
    T = _transform(nside, lmax, nmaps)
    got = T.alm2map(torch.from_numpy(alm).cuda())
    want = osht.alm2map_dense(nside, alm, lmax)
    assert rel(got.cpu().numpy(), want) <= _tol(lmax)
    # map2alm through the adjoint identity <map2alm f, a> = 4 pi / npix <f, alm2map a>
    f = np.random.default_rng(lmax).standard_normal(want.shape)
    back = T.map2alm(torch.from_numpy(f).cuda()).cpu().numpy()
    c = np.where(np.arange(len(alm)) <= lmax, 1.0, 2.0)[:, None]
    lhs = (c * (back * alm.conj()).real).sum(axis=0)
    rhs = 4 * np.pi / (12 * nside * nside) * (f * want).sum(axis=0)
    scale = 4 * np.pi / (12 * nside * nside) * np.linalg.norm(f, axis=0) * np.linalg.norm(want, axis=0)
    assert np.all(np.abs(lhs - rhs) <= _tol(lmax) * scale)
    T.close()


@pytest.mark.parametrize("nside,lmax", [(16, 33), (64, 191)])
@pytest.mark.parametrize("nmaps", [2, 3, 4, 5, 6, 8, 9, 12, 17])
def test_every_map_count_gives_the_same_bits(nside, lmax, nmaps):
    """A map's result does not depend on the maps beside it: the order of
    every sum is the same in each number-of-vectors variant."""
    torch = pytest.importorskip("torch")
    alm = torch.from_numpy(osht.random_alm(lmax, nmaps, seed=nmaps)).cuda()
    T, one = _transform(nside, lmax, nmaps), _transform(nside, lmax, 1)
    maps = T.alm2map(alm)
    back = T.map2alm(maps)
    for k in (0, nmaps // 2, nmaps - 1):
        single = one.alm2map(alm[:, k:k + 1].contiguous())
        assert torch.equal(maps[:, k:k + 1], single)
        assert torch.equal(back[:, k:k + 1], one.map2alm(single))
    T.close()
    one.close()


def test_unaligned_buffers():
    """alm and map pointers of C callers may be 8-byte aligned only."""
    torch = pytest.importorskip("torch")
    from wavemoth_b200 import _native
    nside, lmax, nmaps = 32, 70, 3
    T = _transform(nside, lmax, nmaps)
    alm = torch.from_numpy(osht.random_alm(lmax, nmaps, seed=1)).cuda()
    want = T.alm2map(alm)
    back = T.map2alm(want)
    na, nm = 2 * alm.numel(), want.numel()
    a = torch.zeros(na + 1, dtype=torch.float64, device="cuda")
    a[1:] = torch.view_as_real(alm).reshape(-1)
    m = torch.zeros(nm + 1, dtype=torch.float64, device="cuda")
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    L = _native.lib()
    assert L.wavemoth_execute_alm2map_device(T.plan_handle, a.data_ptr() + 8, m.data_ptr() + 8, stream) == 0
    assert torch.equal(m[1:].reshape(want.shape), want)
    assert L.wavemoth_execute_map2alm_device(T.plan_handle, m.data_ptr() + 8, a.data_ptr() + 8, stream) == 0
    assert torch.equal(a[1:], torch.view_as_real(back).reshape(-1))
    T.close()


@pytest.mark.parametrize("nside,lmax,chunk", [(16, 37, 4), (32, 63, 8), (64, 150, 16)])
def test_depth_one_trees(nside, lmax, chunk):
    """T and B row groups (X buffer rows, blocks that begin inside a group)."""
    torch = pytest.importorskip("torch")
    nmaps, eps = 5, 1e-13
    path = plan_file(nside, lmax, chunk, eps, 1e-10, max_levels=1)
    from wavemoth_b200.sht import Transform
    alm = osht.random_alm(lmax, nmaps, seed=7)
    T = Transform(path, nside, lmax, nmaps)
    got = T.alm2map(torch.from_numpy(alm).cuda())
    back = T.map2alm(got).cpu().numpy()
    f = osht.Rev1File(path)
    want = osht.alm2map_butterfly(f, alm, lmax)
    assert rel(got.cpu().numpy(), want) <= _tol(lmax)
    assert rel(back, osht.map2alm_butterfly(f, got.cpu().numpy(), lmax)) <= _tol(lmax)
    T.close()
