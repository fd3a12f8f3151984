"""Split requests on one image, one with a wait limit: the limit decides the
kernels of a plan of few maps and bounds their waits, so the two do not run as
one transform, and each request's output equals its single call bit for bit."""
import pytest

from oracle import sht as osht
from wavemoth_b200 import _native

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nside,lmax", [(32, 64), (128, 300)])
@pytest.mark.parametrize("limited", [0, 1])
def test_requests_with_different_limits_stay_apart(tmp_path, nside, lmax, limited):
    import torch
    from wavemoth_b200.batch import Batch
    from wavemoth_b200.sht import Transform
    reqs, singles = [], []
    for i, nmaps in enumerate((2, 3, 2)):
        T = Transform(None, nside, lmax, nmaps, precision="split", dense=True)
        if i == limited:
            assert _native.lib().wavemoth_plan_set_wait_limit(T.plan_handle, 1 << 26) == 0
        a = torch.from_numpy(osht.random_alm(lmax, nmaps, seed=i)).cuda()
        out = torch.full((T.npix, nmaps), float("nan"), dtype=torch.float64, device="cuda")
        reqs.append((T, "alm2map", a, out))
        singles.append(T.alm2map(a))
    B = Batch(reqs, cache=str(tmp_path / "schedules.json"))
    assert B.transforms() == 2
    B.execute()
    torch.cuda.synchronize()
    for (T, _, _, out), want in zip(reqs, singles):
        T.device_status()
        assert torch.equal(out, want)
    B.close()
    for r in reqs:
        r[0].close()
