"""What a split-precision image holds, and which kernels its plans run: the
sliced P is made for the first plan of many maps (or with a wait limit), the
FP64 tables for the first of few maps, neither for plans that generate P."""
import pytest

from oracle import sht as osht
from wavemoth_b200 import _native

pytestmark = pytest.mark.gpu

NSIDE, LMAX = 128, 300


def _plan(nmaps, precision="split"):
    from wavemoth_b200.sht import Transform
    return Transform(None, NSIDE, LMAX, nmaps, precision=precision, dense=True)


def _limit(T, polls):
    assert _native.lib().wavemoth_plan_set_wait_limit(T.plan_handle, polls) == 0


def _run(T, nmaps):
    import torch
    f = T.alm2map(torch.from_numpy(osht.random_alm(LMAX, nmaps, seed=nmaps)).cuda())
    a = T.map2alm(f)
    torch.cuda.synchronize()
    T.device_status()
    return f, a


def _same(x, y):
    import torch
    return all(torch.equal(a, b) for a, b in zip(x, y))


def _close(x, y):
    """The split GEMMs keep 42 bits of each operand."""
    return all(float((a - b).abs().max()) <= 1e-10 * float(b.abs().max()) for a, b in zip(x, y))


@pytest.mark.parametrize("few_first", [True, False])
def test_tables_are_made_for_the_plans_that_read_them(few_first):
    alone = {}
    for nmaps in (3, 40):
        T = _plan(nmaps)
        alone[nmaps] = T.work()["image_bytes"]
        T.close()
    G = _plan(3, "split-generate")
    neither = G.work()["image_bytes"]
    assert G.route == "gemm-generate"
    order = (3, 40) if few_first else (40, 3)
    T = {n: _plan(n) for n in order}
    assert T[3].route == "fp64" and T[40].route == "gemm"
    tables, slices = alone[3] - neither, alone[40] - neither
    assert tables > 0 and slices > 0
    assert T[3].work()["image_bytes"] == T[40].work()["image_bytes"] == neither + tables + slices
    D = {n: _plan(n, "double") for n in order}
    for n in order:
        got, want = _run(T[n], n), _run(D[n], n)
        assert _same(got, want) if n == 3 else _close(got, want)
    # the GEMMs on stored slices, on the plan of few maps, give the bits of the generating ones
    _limit(T[3], 1 << 26)
    assert T[3].route == "gemm"
    assert _same(_run(T[3], 3), _run(G, 3))
    _limit(T[3], 0)
    assert T[3].route == "fp64"
    assert _same(_run(T[3], 3), _run(D[3], 3))
    for t in (G, *T.values(), *D.values()):
        t.close()


def test_wait_limit_on_a_plan_of_few_maps_makes_the_slices():
    import torch
    T = _plan(3)
    before = T.work()["image_bytes"]
    x = torch.zeros(4, device="cuda")
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):  # allowed while another stream is captured
        _limit(T, 1 << 26)
        x += 1
    assert T.route == "gemm" and T.work()["image_bytes"] > before
    got = _run(T, 3)
    G = _plan(3, "split-generate")
    assert _same(got, _run(G, 3))
    graph.replay()
    torch.cuda.synchronize()
    assert float(x[0]) == 1.0
    T.close()
    G.close()


def test_without_room_for_the_tables():
    """Under a cap that holds the plan but not its tables it runs the GEMMs,
    generating P; a plan made later, with room, has the tables, and the first
    one's route and results stay."""
    G = _plan(3, "split-generate")
    used = G.work()["device_bytes"]
    want = _run(G, 3)
    G.close()
    L = _native.lib()
    L.wavemoth_set_device_memory_cap(used + (8 << 20))
    try:
        T = _plan(3)
    finally:
        L.wavemoth_set_device_memory_cap(0)
    assert T.route == "gemm-generate"
    assert _same(_run(T, 3), want)
    U, D = _plan(3), _plan(3, "double")
    assert U.route == "fp64" and T.route == "gemm-generate"
    assert _same(_run(U, 3), _run(D, 3)) and _same(_run(T, 3), want)
    for t in (T, U, D):
        t.close()


@pytest.mark.parametrize("precision,nmaps,polls,gemms", [("double", 3, 0, False), ("split", 3, 0, False),
                                                         ("split", 3, 1 << 26, True), ("split", 40, 0, True),
                                                         ("split-generate", 3, 0, True)])
def test_reported_work_is_that_of_the_kernels_that_run(precision, nmaps, polls, gemms):
    T = _plan(nmaps, precision)
    if polls:
        _limit(T, polls)
    work = T.work()
    for key in ("split_int8_ops_alm2map", "split_int8_ops_map2alm", "split_elems_alm2map", "split_elems_map2alm"):
        assert (work[key] > 0) == gemms
    assert work["legendre_flops"] > 0
    T.close()
