"""Gradients of a Transform with ring weights set.  alm2map has no weights: its
gradient, and the adjoint of a bound alm2map plan, equal those without, bit for
bit.  map2alm's are the gradients of a weighted sum over pixels: the unweighted
ones times the pixels' weights, up to a rounding."""
import ctypes

import numpy as np
import pytest

from oracle import sht as osht
from wavemoth_b200 import _native
from wavemoth_b200 import lib as wlib
from wavemoth_b200 import weights as wts

from .plans import plan_file

pytestmark = pytest.mark.gpu

# FP64 kernels (weights of the alm inside them), and the split GEMMs with a separate weighting
PLANS = [(16, 32, 2, "double", True), (32, 64, 3, "double", False), (32, 64, 3, "split", False)]


def _transform(nside, lmax, nmaps, precision, dense):
    from wavemoth_b200.sht import Transform
    return Transform(None if dense else plan_file(nside, lmax, 16, 1e-10, 20.0), nside, lmax, nmaps,
                     precision=precision, dense=dense)


@pytest.mark.parametrize("nside,lmax,nmaps,precision,dense", PLANS)
def test_gradient_of_alm2map(nside, lmax, nmaps, precision, dense):
    torch = pytest.importorskip("torch")
    from wavemoth_b200 import autograd
    T = _transform(nside, lmax, nmaps, precision, dense)
    a = torch.from_numpy(osht.random_alm(lmax, nmaps, seed=1)).cuda().requires_grad_(True)
    g = torch.from_numpy(np.random.default_rng(2).standard_normal((T.npix, nmaps))).cuda()
    (want,) = torch.autograd.grad(autograd.alm2map(a, T), a, g)
    T.set_ring_weights(wts.ring_weights(nside))
    (got,) = torch.autograd.grad(autograd.alm2map(a, T), a, g)
    assert torch.equal(got, want)
    T.close()


def test_adjoint_of_a_bound_alm2map_plan():
    nside, lmax, nmaps = 16, 32, 2
    alm, out = osht.random_alm(lmax, nmaps, seed=3), np.zeros((12 * nside * nside, nmaps))
    P = wlib.ShtPlan(nside, lmax, lmax, alm, out, "mmajor", matrix_data_filename=plan_file(nside, lmax, 8, 1e-10, 1e-10))
    out[:] = np.random.default_rng(4).standard_normal(out.shape)
    want = P.execute_adjoint().copy()
    w = np.ascontiguousarray(wts.ring_weights(nside))
    assert _native.lib().wavemoth_plan_set_ring_weights(P._plan, w.ctypes.data_as(ctypes.POINTER(ctypes.c_double))) == 0
    assert np.array_equal(P.execute_adjoint(), want)
    P.close()


def _pixel_weights(nside, w):
    from wavemoth_b200.healpix import get_ring_offsets
    offs, mid = get_ring_offsets(nside), 2 * nside - 1
    out = np.empty((12 * nside * nside, 1))
    for ring in range(4 * nside - 1):
        out[offs[ring]:offs[ring + 1]] = w[abs(ring - mid)]
    return out


@pytest.mark.parametrize("nside,lmax,nmaps,precision,dense", PLANS[:2])
def test_gradient_of_weighted_map2alm(nside, lmax, nmaps, precision, dense):
    torch = pytest.importorskip("torch")
    from wavemoth_b200 import autograd
    T = _transform(nside, lmax, nmaps, precision, dense)
    f = torch.from_numpy(np.random.default_rng(5).standard_normal((T.npix, nmaps))).cuda().requires_grad_(True)
    b = torch.from_numpy(osht.random_alm(lmax, nmaps, seed=6)).cuda()
    w = wts.ring_weights(nside)
    (plain,) = torch.autograd.grad(autograd.map2alm(f, T), f, b)
    T.set_ring_weights(w)
    out = autograd.map2alm(f, T)
    T.set_ring_weights(None)  # the weights of the forward call count
    (got,) = torch.autograd.grad(out, f, b)
    want = plain.cpu().numpy() * _pixel_weights(nside, w)
    assert np.abs(got.cpu().numpy() - want).max() <= 4e-16 * np.abs(want).max()
    # and the dot product <map2alm(f), b> = <f, grad>
    lhs = float((out.detach().real * b.real + out.detach().imag * b.imag).sum())
    rhs = float((f.detach() * got).sum())
    assert abs(lhs - rhs) <= 1e-12 * float(f.detach().norm() * got.norm())
    T.close()


def test_adjoint_of_a_bound_weighted_map2alm_plan():
    nside, lmax, nmaps = 16, 32, 2
    f = np.random.default_rng(7).standard_normal((12 * nside * nside, nmaps))
    alm = np.zeros(((lmax + 1) * (lmax + 2) // 2, nmaps), np.complex128)
    P = wlib.ShtPlan(nside, lmax, lmax, f, alm, "mmajor", matrix_data_filename=plan_file(nside, lmax, 8, 1e-10, 1e-10),
                     direction="map2alm")
    alm[:] = osht.random_alm(lmax, nmaps, seed=8)
    plain = P.execute_adjoint().copy()
    w = wts.ring_weights(nside)
    assert _native.lib().wavemoth_plan_set_ring_weights(P._plan, w.ctypes.data_as(ctypes.POINTER(ctypes.c_double))) == 0
    got = P.execute_adjoint().copy()
    assert np.array_equal(got, plain * _pixel_weights(nside, w))
    P.close()
