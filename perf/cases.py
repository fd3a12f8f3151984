"""The work whose time this framework is judged by: spherical harmonic
transforms on HEALPix grids through the calls a user's program makes.

A case is a dict of plain values:

  call       what a pass is (see run):
               a2m      Transform.alm2map
               m2a      Transform.map2alm
               trip     alm2map of the batch, then map2alm of that map
               iter     map2alm with ring weights and three Jacobi iterations
               grad     a weighted least-squares loss of alm2map and its gradient
               host     ShtPlan.execute on bound host arrays (the reference's own API)
               batch    one graph launch of several uneven requests
  nside, lmax, nmaps      the grid, the band limit, the maps transformed together
  precision  "double" (the default) or "split"
  plan       "dense"     no plan file: one Legendre recurrence per (m, parity)
             "file"      a plan file as the writer makes it by default
             "levels"    a plan file with one interpolation level everywhere
                         the tree allows it, which is what the writer's
                         choice comes to at nside 1024 and above

`exact` restates the transform with plain torch in 64 bits: the associated
Legendre functions by the three-term recurrence in l with a separate
exponent, one complex FFT per ring length.
"""
import math
import os
import tempfile

import numpy as np
import torch

from wavemoth_b200 import autograd, resource
from wavemoth_b200.batch import Batch
from wavemoth_b200.lib import ShtPlan
from wavemoth_b200.sht import Transform
from wavemoth_b200.weights import ring_weights


def case(name, call, nside, lmax, nmaps, precision="double", plan="dense"):
    return {"name": name, "call": call, "nside": nside, "lmax": lmax, "nmaps": nmaps, "precision": precision,
            "plan": plan}


def listed():
    return [
        # polarisation triplet of a low-resolution analysis, lmax = 3 nside - 1: the smallest call, latency only
        case("m2a 32 x3", "m2a", 32, 95, 3),
        # one sky per call inside a sampler, default plan file
        case("a2m 64 x1", "a2m", 64, 128, 1, plan="file"),
        # analysis as it is usually asked for: quadrature weights and three iterations
        case("iter 128 x3", "iter", 128, 256, 3, plan="file"),
        # differentiable map making: one forward and one backward transform
        case("grad 256 x1", "grad", 256, 512, 1),
        # the reference's own call on host arrays, copies included
        case("host 128 x3", "host", 128, 256, 3, plan="file"),
        # FP64 with interpolation levels, an odd number of maps
        case("trip 256 x7 levels", "trip", 256, 512, 7, plan="levels"),
        # a batch of simulations in split precision with interpolation levels
        case("trip 256 x32 levels split", "trip", 256, 512, 32, "split", "levels"),
        # uneven requests of a serving program in one graph launch
        case("batch 32..128", "batch", 128, 256, 4, "split"),
        # one high-resolution map, FP64
        case("trip 512 x1", "trip", 512, 1024, 1),
        # an ensemble of maps, FP64
        case("trip 512 x16", "trip", 512, 1024, 16),
        # few maps at survey resolution, a band limit that is no power of two
        case("trip 1024 x3 split", "trip", 1024, 1500, 3, "split"),
        # the headline batch: simulations at survey resolution
        case("trip 1024 x32 split", "trip", 1024, 2048, 32, "split"),
    ]


def draw(rng):
    """A case of the same ranges: nside 16 to 1024 (powers of two and a few
    other multiples of 8), lmax from 1.4 to 3 nside - 1, 1 to 32 maps."""
    while True:
        call = rng.choice(["a2m", "m2a", "trip", "trip", "iter", "grad", "host", "batch"])
        lg = rng.uniform(4.0, 10.0)
        nside = 1 << round(lg)
        if nside >= 32 and rng.random() < 0.2:
            nside = 8 * rng.randint(nside // 16 + 1, nside // 8 - 1)
        lmax = rng.randint(int(1.4 * nside), 3 * nside - 1)
        nmaps = round(math.exp(rng.uniform(0.0, math.log(32.0))))
        precision = rng.choice(["double", "split"])
        plan = "dense"
        if nside <= 128 and call != "batch":
            plan = rng.choice(["dense", "file", "levels"])
        if call in ("grad", "host", "iter"):
            nside, nmaps = min(nside, 256 if call == "iter" else 512), min(nmaps, 8)
            lmax = min(lmax, 3 * nside - 1)
        if call == "batch":
            nside, nmaps = min(nside, 256), min(nmaps, 8)
            lmax = min(lmax, 3 * nside - 1)
        c = case("", call, nside, lmax, nmaps, precision, plan)
        del c["name"]
        # no dearer than the ensemble (FP64) or the headline batch (split), and
        # the Legendre matrix no larger than the headline's
        top = listed()[-1 if precision == "split" else -3]
        if work(c)["flops"] <= work(top)["flops"] and lmax * lmax * nside <= 2048 * 2048 * 1024:
            return c


# ---------------------------------------------------------------- inputs

def requests(c):
    """(nside, lmax, nmaps, direction) of every request of a batch case: sizes
    nside / 4, nside / 2 and nside, maps up to nmaps, both directions."""
    out = []
    for i, div in enumerate((4, 4, 2, 2, 1, 1)):
        ns = max(8, c["nside"] // div)
        out.append((ns, min(max(8, c["lmax"] // div), 3 * ns - 1), 1 + (c["nmaps"] - 1) * (i + 1) // 6,
                    "map2alm" if i % 3 == 2 else "alm2map"))
    return out


def random_alm(lmax, nmaps, gen):
    """re/im iid N(0, 1) / (l + 1), imaginary part 0 at m = 0."""
    n = (lmax + 1) * (lmax + 2) // 2
    a = torch.randn((n, nmaps, 2), generator=gen, dtype=torch.float64, device="cuda")
    l = torch.cat([torch.arange(m, lmax + 1) for m in range(lmax + 1)]).cuda()
    a /= (l + 1.0)[:, None, None]
    a[: lmax + 1, :, 1] = 0.0
    return torch.view_as_complex(a)


def random_map(nside, nmaps, gen):
    return torch.randn((12 * nside * nside, nmaps), generator=gen, dtype=torch.float64, device="cuda")


def inputs(c, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(seed)
    if c["call"] == "batch":
        return [random_alm(lm, nm, gen) if d == "alm2map" else random_map(ns, nm, gen)
                for ns, lm, nm, d in requests(c)]
    if c["call"] == "m2a":
        return random_map(c["nside"], c["nmaps"], gen)
    if c["call"] == "iter":
        return random_map(c["nside"], c["nmaps"], gen), ring_weights(c["nside"])
    a = random_alm(c["lmax"], c["nmaps"], gen)
    if c["call"] != "grad":
        return a
    w = 0.5 + torch.rand((12 * c["nside"] ** 2, c["nmaps"]), generator=gen, dtype=torch.float64, device="cuda")
    return a, random_map(c["nside"], c["nmaps"], gen), w


def plan_file(c):
    """Path of the case's plan file, written on first use (a user writes it
    once per (nside, lmax) and keeps it); None for dense plans."""
    if c["plan"] == "dense":
        return None
    folder = os.path.join(tempfile.gettempdir(), "wavemoth_cases_%d" % os.getuid())
    os.makedirs(folder, exist_ok=True)
    path = os.path.join(folder, "%s_%d_%d.dat" % (c["plan"], c["nside"], c["lmax"]))
    if not os.path.exists(path):
        levels = c["plan"] == "levels"
        resource.compute_resource_file(path, c["nside"], c["lmax"], memop_cost=1e-10 if levels else 20.0,
                                       max_workers=1, max_levels=1 if levels else None)
    return path


def prepare(c, seed):
    x = inputs(c, seed)
    s = {"case": c, "x": x}
    nside, lmax, nmaps = c["nside"], c["lmax"], c["nmaps"]
    if c["call"] == "batch":
        reqs = []
        for (ns, lm, nm, d), xi in zip(requests(c), x):
            T = Transform(None, ns, lm, nm, precision=c["precision"], dense=True)
            out = (torch.empty((T.npix, nm), dtype=torch.float64, device="cuda") if d == "alm2map" else
                   torch.empty((T.nalm, nm), dtype=torch.complex128, device="cuda"))
            reqs.append((T, d, xi, out))
        s["outs"] = [r[3] for r in reqs]
        s["batch"] = Batch(reqs, cache=os.path.join(tempfile.gettempdir(), "wavemoth_cases_%d.json" % os.getuid()))
        s["reqs"] = reqs
        return s
    if c["call"] == "host" and c["plan"] != "dense":
        alm = x.cpu().numpy()
        out = np.zeros((12 * nside * nside, nmaps))
        s["plan"] = ShtPlan(nside, lmax, lmax, alm, out, "mmajor", matrix_data_filename=plan_file(c),
                            precision=c["precision"])
        return s
    s["T"] = Transform(plan_file(c), nside, lmax, nmaps, precision=c["precision"], dense=c["plan"] == "dense")
    if c["call"] == "host":
        # the same copies around a plan without a file: pinned host arrays in and out
        s["host_in"] = x.cpu().pin_memory()
        s["host_out"] = torch.empty((12 * nside * nside, nmaps), dtype=torch.float64).pin_memory()
    if c["call"] == "iter":
        s["T"].set_ring_weights(x[1])
    if c["call"] == "grad":
        s["a"] = x[0].clone().requires_grad_(True)
    return s


def run(s):
    c = s["case"]
    call = c["call"]
    if call == "batch":
        s["batch"].execute()
        return s["outs"]
    if "plan" in s:
        return s["plan"].execute()
    T = s["T"]
    if call == "host":
        s["host_out"].copy_(T.alm2map(s["host_in"].cuda(non_blocking=True)), non_blocking=True)
        torch.cuda.current_stream().synchronize()  # the host reads its map
        return s["host_out"]
    if call == "a2m":
        return T.alm2map(s["x"])
    if call == "m2a":
        return T.map2alm(s["x"])
    if call == "iter":
        return T.map2alm(s["x"][0], niter=3)
    if call == "grad":
        _, d, w = s["x"]
        f = autograd.alm2map(s["a"], T)
        loss = (w * (f - d) ** 2).sum()
        (g,) = torch.autograd.grad(loss, s["a"])
        return {"loss": loss.detach(), "map": f.detach(), "grad": g}
    f = T.alm2map(s["x"])
    return [f, T.map2alm(f)]


# ------------------------------------------------------ work and tolerance

def one_way(nside, lmax, nmaps):
    """(bytes, flops) of one direction: alm and map once; a multiply-add per
    (l, m, ring pair, vector) where the Legendre functions are not
    exponentially small (l sin theta >= m), and a real FFT per ring."""
    nalm, npix = (lmax + 1) * (lmax + 2) // 2, 12 * nside * nside
    _, sin = ring_geometry(nside, "cpu")
    elems = float((sin * (nalm + 0.5 * lmax)).sum())
    fft = sum(2.5 * 4 * i * math.log2(4 * i) for i in range(1, nside)) * 2 + \
        (2 * nside + 1) * 2.5 * 4 * nside * math.log2(4 * nside)
    return 16.0 * nalm * nmaps + 8.0 * npix * nmaps, 2.0 * elems * 2 * nmaps + fft * nmaps


def work(c):
    if c["call"] == "batch":
        each = [one_way(ns, lm, nm) for ns, lm, nm, _ in requests(c)]
        return {"bytes": sum(b for b, _ in each), "flops": sum(f for _, f in each)}
    b, f = one_way(c["nside"], c["lmax"], c["nmaps"])
    n = {"trip": 2, "grad": 2, "iter": 7}.get(c["call"], 1)
    return {"bytes": b * n, "flops": f * n}


def tolerance(c):
    """About four times the distance from `exact` measured where the Legendre
    functions carry it: FP64 2.2e-13 at most (recurrences of up to 2048
    steps), split precision 3.5e-12 (42 bits of each operand relative to its
    largest entry).  What a plan file with interpolation levels is off (the
    writer's 1e-10) is common to every implementation that reads it."""
    return {"rel": 1e-12 if c["precision"] == "double" else 1.5e-11}


# ------------------------------------------------------------------ exact

def ring_geometry(nside, device):
    """cos and sin of theta of the 2 nside northern rings, pole first, equator last."""
    i = torch.arange(1, 2 * nside + 1, dtype=torch.float64, device=device)
    h = torch.where(i < nside, i * i / (3.0 * nside * nside), (2.0 * i / nside - 1.0) / 3.0)  # 1 - z
    return 1.0 - h, torch.sqrt(h * (2.0 - h))


class Exact:
    """alm2map and map2alm (4 pi / npix times the adjoint) in 64 bits."""

    def __init__(self, nside, lmax):
        self.nside, self.lmax = nside, lmax
        self.z, self.s = ring_geometry(nside, "cuda")
        nr = 2 * nside
        # lambda_mm = p 2^(256 e), by products over m with the exponent apart
        p = torch.full((nr,), math.sqrt(0.25 / math.pi), dtype=torch.float64, device="cuda")
        e = torch.zeros((nr,), dtype=torch.int32, device="cuda")
        ps, es = [p], [e]
        for m in range(1, lmax + 1):
            p = -p * self.s * math.sqrt((2.0 * m + 1.0) / (2.0 * m))
            small = p.abs() < 2.0 ** -256
            p = torch.where(small, p * 2.0 ** 256, p)
            e = torch.where(small, e - 1, e)
            ps.append(p)
            es.append(e)
        self.p, self.e = torch.stack(ps), torch.stack(es)

    def blocks(self):
        """(m values, index of (m, l = m) in the alm, Lambda[m, l - m, ring]) of consecutive ranges of m."""
        lmax, nr = self.lmax, 2 * self.nside
        m0 = 0
        while m0 <= lmax:
            K = lmax - m0 + 1
            mc = max(1, min(K, int(6e9 / (8.0 * K * nr))))
            m = torch.arange(m0, m0 + mc, device="cuda")
            md = m.double()[:, None]
            L = torch.zeros((mc, K, nr), dtype=torch.float64, device="cuda")
            cur, prev, e = self.p[m0:m0 + mc], torch.zeros((mc, nr), dtype=torch.float64, device="cuda"), \
                self.e[m0:m0 + mc]
            aprev = None
            for k in range(K):
                if k:
                    l = md + k
                    a = torch.sqrt((4.0 * l * l - 1.0) / (l * l - md * md))
                    nxt = a * (self.z * cur - (prev / aprev if k > 1 else 0.0))
                    prev, cur, aprev = cur, nxt, a
                    if k % 8 == 0:
                        big = (e < 0) & (cur.abs() > 2.0 ** 32)
                        cur = torch.where(big, cur * 2.0 ** -256, cur)
                        prev = torch.where(big, prev * 2.0 ** -256, prev)
                        e = torch.where(big, e + 1, e)
                else:
                    aprev = torch.ones_like(md)
                L[:, k] = torch.where(e == 0, cur, torch.where(e == -1, cur * 2.0 ** -256, 0.0))
            L *= (md[:, :, None] + torch.arange(K, device="cuda")[None, :, None] <= lmax)
            yield m0, mc, K, m * (2 * lmax + 3 - m) // 2, L
            m0 += mc

    def gather(self, start, K, nalm):
        return torch.clamp(start[:, None] + torch.arange(K, device="cuda")[None, :], max=nalm - 1)

    def rings(self, t, to_map, other):
        """Between t[m, ring, map] (ring 0 .. 4 nside - 2 from the north) and the map."""
        ns, lmax = self.nside, self.lmax
        m = torch.arange(lmax + 1, device="cuda")
        nrings = 4 * ns - 1
        first, at = [], 0
        for r in range(nrings):
            first.append(at)
            at += 4 * min(r + 1, ns, nrings - r)
        one = torch.ones((), dtype=torch.float64, device="cuda")
        groups = [(4 * i, [i - 1, nrings - i]) for i in range(1, ns)] + [(4 * ns, list(range(ns - 1, 3 * ns)))]
        for n, rs in groups:
            num = [1 if n < 4 * ns or r == ns - 1 else r % 2 for r in rs]
            ang = (m[:, None] * torch.tensor(num, device="cuda")) % (2 * n)
            ph = torch.polar(one, ang.double() * (math.pi / n))[:, :, None]
            pix = (torch.tensor([first[r] for r in rs], device="cuda")[:, None] + torch.arange(n, device="cuda"))
            nm = t.shape[2]
            for g in range(0, nm, 8):
                if to_map:
                    w = t[:, rs, g:g + 8] * ph
                    F = torch.zeros((n,) + tuple(w.shape[1:]), dtype=torch.complex128, device="cuda")
                    F.index_add_(0, m % n, w)
                    f = torch.fft.ifft(F, dim=0, norm="forward").real
                    other[pix.t().reshape(-1), g:g + 8] = f.reshape(-1, f.shape[2])
                else:
                    f = other[pix.t().reshape(-1), g:g + 8].reshape(n, len(rs), -1)
                    F = torch.fft.fft(f.to(torch.complex128), dim=0)
                    t[:, rs, g:g + 8] = F[m % n] * ph.conj()

    def alm2map(self, alm):
        nm, nr = alm.shape[1], 2 * self.nside
        t = torch.empty((self.lmax + 1, 2 * nr - 1, nm), dtype=torch.complex128, device="cuda")
        for m0, mc, K, start, L in self.blocks():
            a = torch.view_as_real(alm[self.gather(start, K, len(alm))]).reshape(mc, K, 2 * nm)
            ev = torch.bmm(L[:, 0::2].transpose(1, 2), a[:, 0::2])
            od = torch.bmm(L[:, 1::2].transpose(1, 2), a[:, 1::2])
            t[m0:m0 + mc, :nr] = torch.view_as_complex((ev + od).reshape(mc, nr, nm, 2))
            t[m0:m0 + mc, nr:] = torch.view_as_complex((ev - od)[:, :-1].flip(1).reshape(mc, nr - 1, nm, 2))
            del L
        t[1:] *= 2.0
        f = torch.empty((12 * self.nside ** 2, nm), dtype=torch.float64, device="cuda")
        self.rings(t, True, f)
        return f

    def map2alm(self, f):
        nm, nr = f.shape[1], 2 * self.nside
        t = torch.empty((self.lmax + 1, 2 * nr - 1, nm), dtype=torch.complex128, device="cuda")
        self.rings(t, False, f)
        t *= math.pi / (3.0 * self.nside ** 2)
        alm = torch.zeros(((self.lmax + 1) * (self.lmax + 2) // 2, nm), dtype=torch.complex128, device="cuda")
        for m0, mc, K, start, L in self.blocks():
            north = t[m0:m0 + mc, :nr]
            south = torch.zeros_like(north)
            south[:, :-1] = t[m0:m0 + mc, nr:].flip(1)
            a = torch.empty((mc, K, 2 * nm), dtype=torch.float64, device="cuda")
            a[:, 0::2] = torch.bmm(L[:, 0::2], torch.view_as_real(north + south).reshape(mc, nr, 2 * nm))
            a[:, 1::2] = torch.bmm(L[:, 1::2], torch.view_as_real(north - south).reshape(mc, nr, 2 * nm))
            a = torch.view_as_complex(a.reshape(mc, K, nm, 2))
            for i in range(mc):
                k = self.lmax - (m0 + i) + 1
                alm[start[i]:start[i] + k] = a[i, :k]
            del L
        return alm


def exact(c, seed):
    x = inputs(c, seed)
    if c["call"] == "batch":
        return [getattr(Exact(ns, lm), d)(xi) for (ns, lm, _, d), xi in zip(requests(c), x)]
    E = Exact(c["nside"], c["lmax"])
    if c["call"] in ("a2m", "host"):
        f = E.alm2map(x)
        return f.cpu() if c["call"] == "host" else f
    if c["call"] == "m2a":
        return E.map2alm(x)
    if c["call"] == "iter":
        # weight of every ring pair (equator first) per pixel
        x, w = x
        ns, wp = c["nside"], []
        for r in range(4 * ns - 1):
            wp.append(np.full(4 * min(r + 1, ns, 4 * ns - 1 - r), w[abs(2 * ns - 1 - r)]))
        wp = torch.from_numpy(np.concatenate(wp)).cuda()[:, None]
        a = E.map2alm(wp * x)
        for _ in range(3):
            a = a + E.map2alm(wp * (x - E.alm2map(a)))
        return a
    if c["call"] == "grad":
        a, d, w = x
        f = E.alm2map(a)
        g = E.map2alm(2.0 * w * (f - d)) * (3.0 * c["nside"] ** 2 / math.pi)
        g[c["lmax"] + 1:] *= 2.0
        g[: c["lmax"] + 1] = g[: c["lmax"] + 1].real.to(g.dtype)
        return {"loss": (w * (f - d) ** 2).sum(), "map": f, "grad": g}
    f = E.alm2map(x)
    return [f, E.map2alm(f)]
