"""Iterative map2alm allocates its buffers at the first call with niter > 0 and
none later, also when a wait limit then sends a split plan of few maps from the
FP64 kernels (which add to the alm in place) to the split GEMMs."""
import pytest

from oracle import sht as osht
from wavemoth_b200 import _native

pytestmark = pytest.mark.gpu


def _limit(T, polls):
    assert _native.lib().wavemoth_plan_set_wait_limit(T.plan_handle, polls) == 0


def test_captured_after_a_change_of_route():
    import torch
    from wavemoth_b200.sht import Transform
    nside, lmax, nmaps = 128, 300, 3
    T = Transform(None, nside, lmax, nmaps, precision="split", dense=True)
    f = T.alm2map(torch.from_numpy(osht.random_alm(lmax, nmaps, seed=1)).cuda())
    first = T.map2alm(f, niter=1)
    assert T.route == "fp64"
    _limit(T, 1 << 26)
    assert T.route == "gemm"
    held = T.work()["device_bytes"]
    out = torch.empty_like(first)
    T.map2alm(f, out=out)  # loads what a first call of a route loads
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        T.map2alm(f, out=out, niter=1)
    graph.replay()
    torch.cuda.synchronize()
    T.device_status()
    assert T.work()["device_bytes"] == held
    assert torch.equal(out, T.map2alm(f, niter=1))
    assert float((out - first).abs().max()) <= 1e-10 * float(first.abs().max())
    _limit(T, 0)
    assert torch.equal(T.map2alm(f, niter=1), first)
    T.close()
