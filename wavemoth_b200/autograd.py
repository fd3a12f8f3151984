"""Differentiable spherical harmonic transforms (torch.autograd.Function).

alm2map is the real-linear map A from the alm (complex128, m-major, the real
and imaginary parts of every (l, m >= 0) entry as independent real variables;
Im a_l0 does not enter) to the RING-ordered map.  The hand-written map2alm
kernels compute the adjoint transform with the weighted inner product of the
real field,

    map2alm = (4 pi / Npix) W^-1 A^T,   W = diag(c_m), c_0 = 1, c_m = 2,

so the gradients of both directions are one call of the other direction's
kernels with a per-m weight (alm2map's is applied by the kernel that writes
the alm: Transform.alm2map_backward; no Legendre values are stored: the backward
pass regenerates them with the same recurrence as the forward pass):

    alm2map backward:  grad_alm = (Npix / 4 pi) c_m map2alm(grad_map)
    map2alm backward:  grad_map = (4 pi / Npix) w_ring alm2map(grad_alm / c_m)

with w_ring the ring weights set on the Transform at the forward call (1 without).

For complex tensors torch expects grad = dL/dRe + i dL/dIm, which is the
componentwise real gradient above.  Im a_l0 gets a zero gradient (the forward
transform ignores it).  The forward definitions follow src/wavemoth.c:1011-1191
(alm2map) and its adjoint; map2alm has no reference implementation.
"""
import math

import numpy as np
import torch

from .healpix import get_ring_pixel_counts
from .sht import Transform


def _m_weights(lmax, device):
    """c_m per alm row of the m-major layout (1 at m = 0, else 2)."""
    w = torch.full(((lmax + 1) * (lmax + 2) // 2,), 2.0, dtype=torch.float64, device=device)
    w[: lmax + 1] = 1.0
    return w


def _pixel_weights(nside, ring_weights, device):
    """(npix, 1) weight of every pixel: that of its ring's pair (equator first)."""
    pair = np.abs(np.arange(4 * nside - 1) - (2 * nside - 1))
    w = torch.from_numpy(np.repeat(ring_weights[pair], get_ring_pixel_counts(nside)))
    return w.to(device)[:, None]


class _Alm2Map(torch.autograd.Function):
    @staticmethod
    def forward(ctx, alm, transform):
        ctx.transform = transform
        return transform.alm2map(alm)

    @staticmethod
    def backward(ctx, grad_map):
        return ctx.transform.alm2map_backward(grad_map), None


class _Map2Alm(torch.autograd.Function):
    @staticmethod
    def forward(ctx, maps, transform):
        ctx.transform = transform
        ctx.ring_weights = getattr(transform, "ring_weights", None)
        return transform.map2alm(maps)

    @staticmethod
    def backward(ctx, grad_alm):
        T = ctx.transform
        w = _m_weights(T.lmax, grad_alm.device)
        g = (grad_alm / w[:, None]).contiguous()
        # Im of m = 0 rows is not an output of map2alm: drop its cotangent
        g[: T.lmax + 1] = g[: T.lmax + 1].real.to(torch.complex128)
        out = T.alm2map(g) * (4.0 * math.pi / T.npix)
        if ctx.ring_weights is not None:
            out = out * _pixel_weights(T.nside, ctx.ring_weights, out.device)
        return out, None


def alm2map(alm, transform):
    """Differentiable alm2map on `transform` (a wavemoth_b200.sht.Transform)."""
    return _Alm2Map.apply(alm, transform)


def map2alm(maps, transform):
    """Differentiable map2alm on `transform`."""
    return _Map2Alm.apply(maps, transform)


class SphericalHarmonics(torch.nn.Module):
    """Module holding one device plan; forward(alm) -> map, inverse(map) -> alm,
    both differentiable."""

    def __init__(self, resource_file, nside, lmax, nmaps=1):
        super().__init__()
        self.transform = Transform(resource_file, nside, lmax, nmaps)

    def forward(self, alm):
        return alm2map(alm, self.transform)

    def inverse(self, maps):
        return map2alm(maps, self.transform)
