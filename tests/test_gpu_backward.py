"""alm2map_backward (the weighted map2alm of the FP64 and of the split route)
against the adjoint of the oracle's dense transform: for re/im as independent
variables, d<w, A a>/da = (npix / 4 pi) c_m map2alm(w), Im a_l0 = 0."""
import numpy as np
import pytest

from oracle import sht as osht
from wavemoth_b200 import _native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nside,lmax,nmaps", [(8, 17, 1), (32, 95, 3), (64, 130, 20)])
@pytest.mark.parametrize("precision", ["double", "split"])
def test_backward_of_alm2map(nside, lmax, nmaps, precision):
    torch = pytest.importorskip("torch")
    from wavemoth_b200.sht import Transform
    T = Transform(None, nside, lmax, nmaps, precision=precision, dense=True)
    if precision == "split":  # keep the split GEMMs and their separate weighting
        assert _native.lib().wavemoth_plan_set_wait_limit(T.plan_handle, 1 << 26) == 0
    w = np.random.default_rng(lmax).standard_normal((T.npix, nmaps))
    want = osht.map2alm_dense(nside, w, lmax) * (T.npix / (4 * np.pi))
    want[lmax + 1:] *= 2.0
    want[: lmax + 1].imag = 0.0
    got = T.alm2map_backward(torch.from_numpy(w).cuda()).cpu().numpy()
    assert np.all(got[: lmax + 1].imag == 0.0)
    # FP64: rounding of lmax / 2 recurrence steps and of both FFTs; split: 42 bits of the largest entry
    tol = 8 * max(lmax, 16) * 2.0 ** -52 if precision == "double" else 1e-10
    assert np.abs(got - want).max() <= tol * np.abs(want).max()
    T.close()
