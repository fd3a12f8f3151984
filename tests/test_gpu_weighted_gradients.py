"""Gradients of a Transform with ring weights set.  alm2map has no weights: its
gradient, and the adjoint of a bound alm2map plan, equal those without, bit for
bit."""
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
