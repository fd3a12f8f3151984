"""Kernels launched to overlap the end of the kernel before them wait for it:
back-to-back calls on one stream, both directions on one plan (q and the X
buffer rewritten by each call), inputs rewritten by torch kernels between
calls, and the same calls captured into a graph, equal calls that are waited
for one by one."""
import pytest

from oracle import sht as osht

from .plans import plan_file

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nside,lmax,nmaps,levels", [(16, 33, 1, False), (32, 95, 3, False), (64, 150, 5, True),
                                                     (128, 256, 16, False)])
@pytest.mark.parametrize("side_stream", [False, True])
def test_back_to_back_calls(nside, lmax, nmaps, levels, side_stream):
    torch = pytest.importorskip("torch")
    from wavemoth_b200.sht import Transform
    path = plan_file(nside, lmax, 16, 1e-12, 1e-10, max_levels=1) if levels else None
    T = Transform(path, nside, lmax, nmaps, dense=path is None)
    alms = [torch.from_numpy(osht.random_alm(lmax, nmaps, seed=s)).cuda() for s in range(4)]
    want = []
    for a in alms:
        f = T.alm2map(a)
        torch.cuda.synchronize()
        b = T.map2alm(f)
        torch.cuda.synchronize()
        want.append((f, b))
    stream = torch.cuda.Stream() if side_stream else torch.cuda.current_stream()
    stream.wait_stream(torch.cuda.current_stream())
    x = torch.empty_like(alms[0])
    with torch.cuda.stream(stream):
        for rep in range(5):
            got = []
            for a in alms:
                x.copy_(a)
                f = T.alm2map(x)
                x.zero_()
                b = T.map2alm(f)
                got.append((f, b))
            for (f, b), (wf, wb) in zip(got, want):
                assert torch.equal(f, wf) and torch.equal(b, wb)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    f, b = torch.empty_like(want[0][0]), torch.empty_like(want[0][1])
    with torch.cuda.graph(graph):
        T.alm2map(x, out=f)
        T.map2alm(f, out=b)
    for a, (wf, wb) in zip(alms, want):
        x.copy_(a)
        graph.replay()
        assert torch.equal(f, wf) and torch.equal(b, wb)
    torch.cuda.synchronize()
    T.close()
