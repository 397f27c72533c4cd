"""The shell sums of the bispectrum (pyl_bk_shell_fill's powers and fields,
pyl_bk_shell_dots) over disjoint, overlapping, nested, empty and out-of-grid shells, and
the in-place deconvolution, against float64 torch.

Tolerances: the sums' terms are formed and added in float64 by both (1e-12 of the sum of
their sizes); the deconvolved mode rounds its factor, product (and the interlaced
combination) a few times in float32 (2^-20 of the parts' sizes)."""
import ctypes
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


def k2_of(n):
    k = freqs(n)
    return k[:, None, None] ** 2 + k[None, :, None] ** 2 + torch.arange(n // 2 + 1, device='cuda')[None, None, :] ** 2


SHELLS = [(1, 4), (2, 9), (9, 30), (0, 1), (5, 5), (4, 30), (25, 26)]


@pytest.mark.parametrize('dims,side,extra', [(16, 16, [(30, 10 ** 9), (200, 400)]), (15, 15, [(0, 10 ** 9)]),
                                             (64, 18, []), (65, 20, [(7, 8)]), (130, 130, [(900, 1300), (4225, 4226)])])
def test_shell_sums_equal_float64(lib, dims, side, extra):
    from pylians_gb300._device import ptr, stream_ptr
    g = torch.Generator(device='cuda')
    g.manual_seed(dims)
    shells = SHELLS + extra
    n = len(shells)
    lo, hi = [(ctypes.c_int64 * n)(*[s[a] for s in shells]) for a in (0, 1)]
    slots = [0, -1, 2, 1] + [-1] * (n - 4)
    slot, dst = (ctypes.c_int * n)(*slots), (ctypes.c_int * n)(*reversed(range(n)))
    dk = torch.randn((dims, dims, dims // 2 + 1), dtype=torch.complex64, generator=g, device='cuda')
    half = (side, side, side // 2 + 1)
    ph = torch.randn(half, dtype=torch.complex64, generator=g, device='cuda')
    cast = lambda a: ctypes.cast(a, ctypes.c_void_p)
    n2 = k2_of(dims)
    kz = torch.arange(dims // 2 + 1, device='cuda')
    w = torch.where((kz == 0) | (2 * kz == dims), 1.0, 2.0).double().expand(dims, dims, -1)
    p2 = w * (dk.real.double() ** 2 + dk.imag.double() ** 2)
    # the same modes on the side^3 half grid: kx, ky wrapped, kz alike
    k = freqs(dims).remainder(side)
    fits = (freqs(dims).abs() <= side // 2)
    for source, fields in ((dk, (True, False)), (dk, (True, True)), (None, (False, True))):
        power = torch.full((2 * n,), 7.0, dtype=torch.float64, device='cuda')
        od = torch.full((3,) + half, 9.0, dtype=torch.complex64, device='cuda')
        oi = torch.full((3,) + half, 9.0, dtype=torch.complex64, device='cuda')
        lib.call('pyl_bk_shell_fill', ptr(source), dims, side, cast(lo), cast(hi), cast(slot), n,
                 ptr(od) if fields[0] else None, ptr(oi) if fields[1] else None, ptr(power), stream_ptr())
        out = power.cpu().numpy()
        for s, (a, b) in enumerate(shells):
            m = (n2 >= a) & (n2 < b)
            ref = float(p2[m].sum()) if source is not None else 0.0
            assert abs(out[2 * s] - ref) <= 1e-12 * ref and out[2 * s + 1] == float(w[m].sum()), (s, out[2 * s:2 * s + 2])
            if slots[s] < 0:
                continue
            want = torch.zeros((2,) + half, dtype=torch.complex64, device='cuda')
            i, j, l = torch.nonzero(m, as_tuple=True)
            want[0, k[i], k[j], l] = dk[i, j, l]
            want[1, k[i], k[j], l] = 1.0
            for f, got in enumerate((od, oi)):
                if fields[f]:
                    assert torch.equal(got[slots[s]], want[f])
    for source in (dk, None):
        out = torch.full((n,), 0.5, dtype=torch.float64, device='cuda')
        lib.call('pyl_bk_shell_dots', ptr(source), dims, ptr(ph), side, cast(lo), cast(hi), cast(dst), n, ptr(out),
                 stream_ptr())
        got = out.cpu().numpy()
        for s, (a, b) in enumerate(shells):
            m = (n2 >= a) & (n2 < b) & fits[:, None, None] & fits[None, :, None]
            i, j, l = torch.nonzero(m, as_tuple=True)
            v = dk[i, j, l].to(torch.complex128) if source is not None else torch.ones(len(i), dtype=torch.complex128, device='cuda')
            q = ph[k[i], k[j], l].to(torch.complex128)
            ws = torch.where((l == 0) | (2 * l == side), 1.0, 2.0).double()
            t = ws * (v.real * q.real + v.imag * q.imag) / side ** 3
            assert abs(got[n - 1 - s] - 0.5 - float(t.sum())) <= 1e-12 * (float(t.abs().sum()) + 0.5), s


@pytest.mark.parametrize('inter', [False, True])
@pytest.mark.parametrize('dims,p', [(2, 2), (3, 1), (16, 4), (33, 3), (66, 2)])
def test_deconvolve_equals_float64(lib, dims, p, inter):
    from pylians_gb300._device import ptr, stream_ptr
    g = torch.Generator(device='cuda')
    g.manual_seed(dims)
    shape = (dims, dims, dims // 2 + 1)
    dk = torch.randn(shape, dtype=torch.complex64, generator=g, device='cuda')
    dk2 = torch.randn(shape, dtype=torch.complex64, generator=g, device='cuda') if inter else None
    k = freqs(dims)
    t = math.pi * k.double() / dims
    c = torch.where(k == 0, torch.ones_like(t), (t / torch.sin(t)) ** p)
    f = c[:, None, None] * c[None, :, None] * c[None, None, :shape[2]]
    d, size = dk.to(torch.complex128), dk.abs().double()
    if inter:
        s = (k[:, None, None] + k[None, :, None] + torch.arange(shape[2], device='cuda')[None, None, :]).double()
        d = 0.5 * (d + dk2.to(torch.complex128) * torch.polar(torch.ones_like(s), s * (math.pi / dims)))
        size = size + dk2.abs().double()
    lib.call('pyl_mas_deconvolve', ptr(dk), ptr(dk2), dims, p, stream_ptr())
    assert bool(((dk.to(torch.complex128) - d * f).abs() <= 2.0 ** -20 * size * f).all())
