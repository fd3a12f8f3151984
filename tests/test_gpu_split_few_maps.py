"""Split plans of few maps on the FP64 units: every call that reaches their
Legendre step -- both directions, iterated map2alm (the sum inside the kernel),
the gradient of alm2map (the per-m weights inside it) -- on dense images, on files
with interpolation levels and on files with deeper trees, whose generic kernels
leave sum and weights to kernels of their own.  The FP64 plan of the same file
runs the same kernels on the same tables: equal bits."""
import pytest

from oracle import sht as osht

from .plans import plan_file

pytestmark = pytest.mark.gpu

# nside, lmax, chunk size (None: dense), levels allowed; at least 2^22 recurrence elements each
IMAGES = [(128, 300, None, None), (128, 300, 16, 1), (128, 383, 64, 1), (128, 383, 16, 2)]


@pytest.mark.parametrize("nside,lmax,chunk,levels", IMAGES)
@pytest.mark.parametrize("nmaps", [1, 3, 14])
def test_equal_to_the_fp64_plan(nside, lmax, chunk, levels, nmaps):
    torch = pytest.importorskip("torch")
    from wavemoth_b200 import weights as wts
    from wavemoth_b200.sht import Transform
    path = plan_file(nside, lmax, chunk, 1e-12, 1e-10, workers=8, max_levels=levels) if chunk else None
    alm = torch.from_numpy(osht.random_alm(lmax, nmaps, seed=nmaps)).cuda()
    out = {}
    for precision in ("split", "double"):
        T = Transform(path, nside, lmax, nmaps, precision=precision, dense=path is None)
        assert T.route == "fp64"
        f = T.alm2map(alm)
        got = [f, T.map2alm(f), T.alm2map_backward(f)]
        T.set_ring_weights(wts.ring_weights(nside))
        got += [T.map2alm(f), T.map2alm(f, niter=2)]
        torch.cuda.synchronize()
        T.device_status()
        out[precision] = got
        T.close()
    for got, want in zip(out["split"], out["double"]):
        assert bool(torch.isfinite(torch.view_as_real(want) if want.is_complex() else want).all())
        assert torch.equal(got, want)


@pytest.mark.parametrize("nside,lmax,chunk,levels", IMAGES[1:])
def test_interpolation_levels_against_the_dense_transform(nside, lmax, chunk, levels):
    """Files of precision 1e-12: an interpolative decomposition of k out of n
    columns errs by up to sqrt(1 + k (n - k)) eps, 7e-11 for n = 128; two levels
    twice that."""
    torch = pytest.importorskip("torch")
    from wavemoth_b200.sht import Transform
    path = plan_file(nside, lmax, chunk, 1e-12, 1e-10, workers=8, max_levels=levels)
    alm = torch.from_numpy(osht.random_alm(lmax, 2, seed=3)).cuda()
    S = Transform(path, nside, lmax, 2, precision="split")
    D = Transform(None, nside, lmax, 2, dense=True)
    f = D.alm2map(alm)
    for got, want in ((S.alm2map(alm), f), (S.map2alm(f), D.map2alm(f))):
        assert float((got - want).norm()) <= 1.5e-10 * float(want.norm())
    S.close()
    D.close()
