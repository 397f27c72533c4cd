"""The mode and separation kernels of Xi and correct_MAS (sign rows of a representative
at once) against float64 torch, at the edges of their runs and segments along z, where
the mirrored halves of a row meet (odd and even grids), and on grids that lie wholly
inside the small bins.

Tolerances: xi_power and correct_mas round the factor, its product and the square once
each, so within 2^-21 of each value; a bin's float32 sums are chains of at most 2^16
additions, off by 2^8 ulps of the sum of sizes (256 * 2^-24); counts are exact; sums of
|r| are float64 sums of terms good to 2^-47 in another order (1e-12)."""
import math

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope='module')
def lib():
    import pylians_gb300.build as b
    b.build()
    from pylians_gb300 import _lib
    return _lib


def freqs(n):
    k = torch.arange(n, device='cuda')
    return torch.where(k > n // 2, k - n, k)


@pytest.mark.parametrize('dims,axis', [(2, 0), (3, 2), (16, 1), (30, 2), (31, 0), (33, 1), (62, 2), (63, 0), (64, 2), (65, 0),
                                       (130, 1), (290, 2), (578, 0)])
def test_xi_bin_equals_float64(lib, dims, axis):
    from pylians_gb300._device import ptr, stream_ptr
    g = torch.Generator(device='cuda')
    g.manual_seed(dims)
    x = torch.randn((dims,) * 3, generator=g, device='cuda')
    n = lib.load().pyl_xi_sums_len(dims)
    out = torch.full((n,), 7.0, dtype=torch.float64, device='cuda')
    lib.call('pyl_xi_bin', ptr(x), dims, axis, ptr(out), stream_ptr())
    nb = n // 5
    o = out.cpu().numpy()
    r = freqs(dims)
    X, S = np.zeros((nb, 3)), np.zeros((nb, 3))
    R, N = np.zeros(nb), np.zeros(nb)
    for i in range(dims):               # a plane at a time
        r2 = (r[i] ** 2 + r[:, None] ** 2 + r[None, :] ** 2).reshape(-1)
        par = (r[i].expand(dims, dims), r[:, None].expand(dims, dims), r[None, :].expand(dims, dims))[axis].reshape(-1)
        mu2 = torch.where(r2 > 0, par.double() ** 2 / r2.clamp_min(1).double(), 0.0)
        length = torch.sqrt(r2.double())
        b = torch.floor(length).long()
        v = x[i].double().reshape(-1)
        for l, w in enumerate((torch.ones_like(mu2), 0.5 * (3 * mu2 - 1), 0.125 * ((35 * mu2 - 30) * mu2 + 3))):
            X[:, l] += torch.bincount(b, v * w, nb).cpu().numpy()
            S[:, l] += torch.bincount(b, (v * w).abs(), nb).cpu().numpy()
        R += torch.bincount(b, length, nb).cpu().numpy()
        N += torch.bincount(b, minlength=nb).cpu().numpy()
    assert np.array_equal(o[4 * nb:], N)
    np.testing.assert_allclose(o[3 * nb:4 * nb], R, rtol=1e-12)
    assert np.all(np.abs(o[:3 * nb].reshape(nb, 3) - X) <= 256 * 2.0 ** -24 * np.maximum(S, S[:, :1]))


@pytest.mark.parametrize('dims,p', [(2, 2), (3, 4), (16, 3), (33, 1), (130, 2), (131, 0)])
def test_mode_factors_equal_float64(lib, dims, p):
    from pylians_gb300._device import ptr, stream_ptr
    g = torch.Generator(device='cuda')
    g.manual_seed(dims)
    dk = torch.randn((dims, dims, dims // 2 + 1), dtype=torch.complex64, generator=g, device='cuda')
    k = freqs(dims)
    t = math.pi * k.double() / dims
    c = torch.where(k == 0, torch.ones_like(t), (t / torch.sin(t)) ** p)
    f = c[:, None, None] * c[None, :, None] * c[None, None, :dims // 2 + 1]
    d = dk.to(torch.complex128) * f
    power = dk.clone()
    lib.call('pyl_xi_power', ptr(power), dims, p, stream_ptr())
    ref = d.real ** 2 + d.imag ** 2
    assert bool(((power.real.double() - ref).abs() <= 2.0 ** -21 * ref).all()) and not bool(power.imag.any())
    out = dk.clone()
    lib.call('pyl_correct_mas', ptr(out), dims, p, stream_ptr())
    kz = torch.arange(dims // 2 + 1, device='cuda')
    inner = (kz != 0) & ((kz != dims // 2) | (dims % 2 == 1))      # the other planes keep their Hermitian part
    err = (out.to(torch.complex128) - d)[..., inner].abs()
    assert bool((err <= 2.0 ** -21 * d[..., inner].abs()).all())


@pytest.mark.parametrize('dims,axis', [(255, 0), (256, 2), (257, 0), (257, 1), (257, 2), (291, 1), (579, 0)])
def test_xi_bin_equals_float64_on_larger_sides(lib, dims, axis):
    test_xi_bin_equals_float64(lib, dims, axis)


@pytest.mark.parametrize('dims', [64, 255, 256, 257, 300])
def test_xi_bin_adds_x_planes_in_float64(lib, dims):
    """2^24 at (x, y, z) and 1 at (-x, y, z), alone in their bins: the float32 sum of the two
    loses the 1, the float64 sum of different x planes is exact."""
    from pylians_gb300._device import ptr, stream_ptr
    x = torch.zeros((dims,) * 3, device='cuda')
    bins = []
    for i in range(4, dims // 2 - 1, 5):
        x[i, 3, 2] = 2.0 ** 24
        x[dims - i, 3, 2] = 1.0
        bins.append(math.isqrt(i * i + 13))
    assert len(set(bins)) == len(bins)
    out = torch.empty(lib.load().pyl_xi_sums_len(dims), dtype=torch.float64, device='cuda')
    lib.call('pyl_xi_bin', ptr(x), dims, 2, ptr(out), stream_ptr())
    got = out.cpu().numpy()[:3 * (len(out) // 5)].reshape(-1, 3)[bins, 0]
    assert np.array_equal(got, np.full(len(bins), 2.0 ** 24 + 1.0))


@pytest.mark.parametrize('dims', [16, 33, 256, 257])
def test_xi_bin_lengths_are_float64(lib, dims):
    """Sums of |r| of the smallest bins: correctly rounded roots (2^-53) and at most one
    rounding for each of a bin's separations."""
    from pylians_gb300._device import ptr, stream_ptr
    x = torch.zeros((dims,) * 3, device='cuda')
    out = torch.empty(lib.load().pyl_xi_sums_len(dims), dtype=torch.float64, device='cuda')
    lib.call('pyl_xi_bin', ptr(x), dims, 0, ptr(out), stream_ptr())
    nb = len(out) // 5
    R = out.cpu().numpy()[3 * nb:4 * nb]
    m = range(-4, 5)
    n2 = [a * a + b * b + c * c for a in m for b in m for c in m]
    for b in (1, 2, 3):
        terms = [math.sqrt(v) for v in n2 if b * b <= v < (b + 1) ** 2]
        ref = math.fsum(terms)
        assert abs(R[b] - ref) <= (len(terms) + 1) * 2.0 ** -53 * ref
