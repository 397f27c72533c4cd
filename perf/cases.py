"""Performance cases of the density-field and clustering path.

Each case is one call (or one short chain of calls) that an analysis makes on a
simulation box of 1000 Mpc/h: mass assignment in its forms (resident tensors and
host arrays, plain and interlaced, masses, the deterministic strategy), the grid
read back at particle positions, power and cross power spectra, the correlation
function, the bispectrum, a batch of realizations, and the whole chain from
particles to P(k).  prepare() makes a program's inputs from the seed with torch
alone, run() is the call, exact() the same quantities in float64 with torch alone.
"""
import math

import numpy as np
import torch

import pylians_gb300.MAS_library as MASL
import pylians_gb300.Pk_library as PKL
from pylians_gb300.batch import RealizationBatch
from pylians_gb300.pipeline import ParticlePk

BOX = 1000.0
SUPPORT = {'NGP': 1, 'CIC': 2, 'TSC': 3, 'PCS': 4}
LINES_OF_SIGHT = (0, 1, 2)


# ------------------------------------------------------------------------ cases
def listed():
    return [
        # the smallest call: a sparse halo catalogue onto a coarse grid, resident
        dict(name='ma_cic_64', kind='ma', dims=64, side=46, mas='CIC', interlaced=False, masses=False,
             strategy='auto', order='random', host=False),
        # a whole simulation snapshot (512^3 lattice-ordered particles) onto 512^3 with
        # the highest-order scheme and interlacing, the input of a precise P(k)
        dict(name='ma_pcs_interlaced_512', kind='ma', dims=512, side=512, mas='PCS', interlaced=True, masses=False,
             strategy='auto', order='lattice', host=False),
        # masses spread over decades (haloes, gas cells) onto a grid that is no
        # multiple of any tile
        dict(name='ma_tsc_masses_500', kind='ma', dims=500, side=300, mas='TSC', interlaced=False, masses=True,
             strategy='auto', order='random', host=False),
        # the drop-in call of the reference's users: numpy positions into a numpy grid
        dict(name='ma_cic_host_256', kind='ma', dims=256, side=256, mas='CIC', interlaced=False, masses=False,
             strategy='auto', order='lattice', host=True),
        # the deterministic strategy (bit-reproducible grids)
        dict(name='ma_tsc_sorted_256', kind='ma', dims=256, side=256, mas='TSC', interlaced=False, masses=False,
             strategy='sorted', order='random', host=False),
        # overdensity at the positions of a catalogue
        dict(name='interp_512', kind='interp', dims=512, side=256, order='random'),
        # P(k) of a small field: one call of many in a loop over snapshots or mocks
        dict(name='pk_128', kind='pk', dims=128, mas='CIC', axis=0, interlaced=False),
        # auto and cross spectra of two tracers in redshift space
        dict(name='xpk_2_512', kind='xpk', dims=512, fields=2, axis=2),
        # correlation function multipoles of a field
        dict(name='xi_256', kind='xi', dims=256, mas='CIC', axis=2),
        # bispectrum over the angle between two sides
        dict(name='bk_256', kind='bk', dims=256, mas='CIC', bins=32),
        # realizations of uneven sizes, schemes and interlacing in one batch
        dict(name='batch_24', kind='batch', count=24, specs=3, axis=0),
        # the whole chain at the largest size: 1024^3 particles onto 1024^3, interlaced
        dict(name='particles_pk_1024', kind='chain', dims=1024, side=1024, mas='CIC', axis=0, interlaced=True,
             order='random'),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(('ma', 'ma', 'ma', 'interp', 'pk', 'xpk', 'xi', 'bk', 'batch', 'chain'))
    mas = rng.choice(('CIC', 'TSC', 'PCS'))
    axis = rng.choice(LINES_OF_SIGHT)
    if kind == 'ma':
        host = rng.random() < 0.2
        strategy = 'sorted' if not host and rng.random() < 0.25 else 'auto'
        big = 256 if host or strategy == 'sorted' else 512
        return dict(kind='ma', dims=_log(rng, 64, big), side=_log(rng, 46, big), mas=rng.choice(('NGP', mas)),
                    interlaced=not host and rng.random() < 0.5, masses=rng.random() < 0.4, strategy=strategy,
                    order=rng.choice(('random', 'lattice')), host=host)
    if kind == 'interp':
        return dict(kind='interp', dims=_log(rng, 64, 512), side=_log(rng, 46, 320),
                    order=rng.choice(('random', 'lattice')))
    if kind == 'pk':
        return dict(kind='pk', dims=_log(rng, 64, 640), mas=mas, axis=axis, interlaced=rng.random() < 0.5)
    if kind == 'xpk':
        return dict(kind='xpk', dims=_log(rng, 64, 512), fields=rng.choice((2, 3, 4)), axis=axis)
    if kind == 'xi':
        return dict(kind='xi', dims=_log(rng, 64, 512), mas=mas, axis=axis)
    if kind == 'bk':
        return dict(kind='bk', dims=_log(rng, 96, 320), mas=mas, bins=_log(rng, 8, 40))
    if kind == 'batch':
        return dict(kind='batch', count=_log(rng, 4, 48), specs=rng.randrange(1 << 20), axis=axis)
    return dict(kind='chain', dims=_log(rng, 64, 768), side=_log(rng, 64, 768), mas=mas, axis=axis,
                interlaced=rng.random() < 0.5, order=rng.choice(('random', 'lattice')))


def _specs(case):
    """Realizations of a batch: grid side, particle count (log-uniform), scheme and
    interlacing of each, from the case's own number."""
    r = np.random.default_rng(case['specs'])
    out = []
    for _ in range(case['count']):
        n = int(math.exp(r.uniform(math.log(1e5), math.log(1.7e7))))
        out.append(dict(dims=int(r.choice((64, 128, 192, 256))), MAS=str(r.choice(('CIC', 'TSC', 'PCS'))),
                        interlaced=bool(r.integers(0, 2)), n=n))
    return out


def _schemes(case):
    return ['TSC', 'CIC', 'NGP', 'PCS'][:case['fields']]


def _triangles(case):
    """Two sides at a quarter and half of the Nyquist wave number, the angle between
    them swept over (0, pi)."""
    kn = math.pi * case['dims'] / BOX
    return 0.25 * kn, 0.5 * kn, np.linspace(0.0, math.pi, case['bins'] + 1)[:-1]


# ----------------------------------------------------------------------- inputs
def _device():
    return torch.device('cuda', torch.cuda.current_device())


def _generator(seed, k=0):
    g = torch.Generator(device=_device())
    g.manual_seed(int(seed) * 1000003 + k)
    return g


def _modes(n, box=BOX, dtype=torch.float32):
    kf = 2.0 * math.pi / box
    k = torch.fft.fftfreq(n, d=1.0 / n, device=_device(), dtype=dtype) * kf
    return k, torch.arange(n // 2 + 1, device=_device(), dtype=dtype) * kf


def _field(n, g, rms=0.5):
    """A Gaussian overdensity field with P(k) ~ k^-1.5 exp(-(k / 0.5)^2) and some shot noise."""
    d = torch.fft.rfftn(torch.randn((n, n, n), generator=g, device=_device()))
    k, kz = _modes(n)
    k2 = k[:, None, None] ** 2 + k[None, :, None] ** 2 + kz[None, None, :] ** 2
    k2[0, 0, 0] = 1.0
    d *= torch.sqrt(k2 ** -0.75 * torch.exp(-k2 / 0.25))
    d[0, 0, 0] = 0.0
    x = torch.fft.irfftn(d, s=(n, n, n))
    x *= rms / x.std()
    x += 0.2 * torch.randn((n, n, n), generator=g, device=_device())
    return x - x.mean()


def _particles(side, g, order):
    """side^3 positions in [0, BOX): uniform in random order, or a lattice in cell
    order moved by a smooth displacement of 4 Mpc/h rms per axis."""
    n = side ** 3
    if order == 'random':
        p = torch.rand((n, 3), generator=g, device=_device()) * BOX
    else:
        m = 64
        k, kz = _modes(m)
        k2 = k[:, None, None] ** 2 + k[None, :, None] ** 2 + kz[None, None, :] ** 2
        k2[0, 0, 0] = 1.0
        d = torch.fft.rfftn(torch.randn((m, m, m), generator=g, device=_device())) * k2 ** -1.375
        d[0, 0, 0] = 0.0
        axis = (torch.arange(side, device=_device(), dtype=torch.float32) + 0.5) * (BOX / side)
        p = torch.empty((side, side, side, 3), device=_device())
        for a, ka in enumerate((k[:, None, None], k[None, :, None], kz[None, None, :])):
            psi = torch.fft.irfftn(1j * ka * d, s=(m, m, m))
            psi *= 4.0 / psi.std()
            p[..., a] = torch.nn.functional.interpolate(psi[None, None], size=(side,) * 3, mode='trilinear',
                                                        align_corners=False)[0, 0]
            p[..., a] += axis.reshape([-1 if b == a else 1 for b in range(3)])
        p = p.reshape(n, 3).remainder_(BOX)
    p[p >= BOX] = 0.0
    return p


def prepare(case, seed):
    g = _generator(seed)
    kind = case['kind']
    if kind == 'ma':
        pos = _particles(case['side'], g, case['order'])
        w = torch.exp(torch.randn(pos.shape[0], generator=g, device=_device())) if case['masses'] else None
        if case['host']:
            pos, w = pos.cpu().numpy(), None if w is None else w.cpu().numpy()
        return dict(case=case, pos=pos, w=w)
    if kind == 'interp':
        return dict(case=case, field=_field(case['dims'], g), pos=_particles(case['side'], g, case['order']))
    if kind in ('pk', 'xi', 'bk'):
        d = _field(case['dims'], g)
        other = d + 0.02 * torch.randn(d.shape, generator=g, device=_device()) if case.get('interlaced') else None
        return dict(case=case, delta=d, other=other)
    if kind == 'xpk':
        d = _field(case['dims'], g)
        return dict(case=case, fields=[d + 0.3 * torch.randn(d.shape, generator=g, device=_device())
                                       for _ in range(case['fields'])])
    if kind == 'batch':
        specs = _specs(case)
        # work items of the default size, so that a pass does not depend on a timing
        return dict(case=case, batch=RealizationBatch(specs, BOX, axis=case['axis'], tune=False),
                    pos=[torch.rand((s['n'], 3), generator=g, device=_device()) * (BOX * (1 - 1e-6)) for s in specs])
    pos = _particles(case['side'], g, case['order'])
    return dict(case=case, pos=pos, plan=ParticlePk(case['dims'], BOX, case['mas'], axis=case['axis'],
                                                    interlaced=case['interlaced'], max_particles=pos.shape[0]))


# ------------------------------------------------------------------------- pass
def run(state):
    case = state['case']
    kind, dims = case['kind'], case.get('dims')
    if kind == 'ma':
        if case['host']:
            delta = np.zeros((dims,) * 3, dtype=np.float32)
            MASL.MA(state['pos'], delta, BOX, case['mas'], state['w'])
            return delta
        delta = torch.zeros((dims,) * 3, device=_device())
        shifted = torch.zeros((dims,) * 3, device=_device()) if case['interlaced'] else None
        MASL.MA(state['pos'], delta, BOX, case['mas'], state['w'], interlaced=shifted, strategy=case['strategy'])
        return [delta] if shifted is None else [delta, shifted]
    if kind == 'interp':
        den = torch.empty(state['pos'].shape[0], device=_device())
        MASL.CIC_interp(state['field'], BOX, state['pos'], den)
        return den
    if kind == 'pk':
        return _attributes(PKL.Pk(state['delta'], BOX, case['axis'], case['mas'], interlaced=state['other']))
    if kind == 'xpk':
        return _attributes(PKL.XPk(state['fields'], BOX, case['axis'], _schemes(case)))
    if kind == 'xi':
        return _attributes(PKL.Xi(state['delta'], BOX, case['mas'], case['axis']))
    if kind == 'bk':
        k1, k2, theta = _triangles(case)
        return _attributes(PKL.Bk(state['delta'], BOX, k1, k2, theta, case['mas']))
    if kind == 'batch':
        state['batch'].step(state['pos'])
        return state['batch'].sums
    state['plan'].step(state['pos'])
    return _attributes(state['plan'].result())


def _attributes(result):
    return {k: v for k, v in vars(result).items() if isinstance(v, np.ndarray)}


# ------------------------------------------------------------------------- work
def work(case):
    """Inputs read once, outputs written once, and the arithmetic of the transforms
    (2.5 N log2 N a real transform) and of the weights and sums."""
    kind = case['kind']
    if kind == 'batch':
        b = f = 0
        for s in _specs(case):
            x = work(dict(kind='chain', dims=s['dims'], n=s['n'], mas=s['MAS'], interlaced=s['interlaced']))
            b, f = b + x['bytes'], f + x['flops']
        return dict(bytes=b, flops=f)
    d = case['dims']
    cells, modes = d ** 3, d * d * (d // 2 + 1)
    bins = 8.0 * (0.36 * d * d + 5 * d)
    fft = 2.5 * cells * math.log2(cells)
    if kind in ('ma', 'chain'):
        n = case.get('n') or case['side'] ** 3
        grids = 2 if case['interlaced'] else 1
        s = SUPPORT[case['mas']]
        flops = n * grids * (8.0 * s + 2.0 * s ** 3)
        if kind == 'ma':
            return dict(bytes=n * (16.0 if case['masses'] else 12.0) + 4.0 * grids * cells, flops=flops)
        return dict(bytes=12.0 * n + bins, flops=flops + grids * (fft + 40.0 * modes))
    if kind == 'interp':
        n = case['side'] ** 3
        return dict(bytes=4.0 * cells + 16.0 * n, flops=40.0 * n)
    if kind == 'pk':
        grids = 2 if case['interlaced'] else 1
        return dict(bytes=4.0 * grids * cells + bins, flops=grids * (fft + 40.0 * modes))
    if kind == 'xpk':
        nf = case['fields']
        return dict(bytes=4.0 * nf * cells + bins * nf * (nf + 1) / 2, flops=nf * fft + 20.0 * nf * (nf + 1) * modes)
    if kind == 'xi':
        return dict(bytes=4.0 * cells + 40.0 * d, flops=2 * fft + 20.0 * modes + 20.0 * cells)
    return dict(bytes=4.0 * cells + 64.0 * case['bins'], flops=fft + 20.0 * modes + case['bins'] * 8.0 * modes)


# ---------------------------------------------------------------- float64 values
EXACT_ADDS = 1.2e10          # corner additions that take some ten seconds in float64


def _weights(x, mas):
    """First cell and the weights along one axis of float64 grid coordinates."""
    if mas == 'NGP':
        return torch.floor(x + 0.5).long(), [torch.ones_like(x)]
    if mas == 'CIC':
        f = torch.floor(x)
        u = x - f
        return f.long(), [1.0 - u, u]
    if mas == 'TSC':
        f = torch.floor(x - 0.5)
        u = x - f - 1.0                         # distance to the middle cell, [-1/2, 1/2)
        return f.long(), [0.5 * (0.5 - u) ** 2, 0.75 - u * u, 0.5 * (0.5 + u) ** 2]
    f = torch.floor(x) - 1.0
    out = []
    for j in range(4):
        s = (x - f - j).abs()
        out.append(torch.where(s < 1.0, (4.0 - 6.0 * s * s + 3.0 * s ** 3) / 6.0,
                               (2.0 - s).clamp_min(0.0) ** 3 / 6.0))
    return f.long(), out


def _deposit(pos, w, dims, mas, shift):
    grid = torch.zeros(dims ** 3, dtype=torch.float64, device=_device())
    step = 1 << 23
    for i in range(0, pos.shape[0], step):
        x = pos[i:i + step].double() * (dims / BOX) + shift
        axes = [_weights(x[:, a], mas) for a in range(3)]
        m = None if w is None else w[i:i + step].double()
        for l, wx in enumerate(axes[0][1]):
            ix = (axes[0][0] + l).remainder(dims) * dims
            for k, wy in enumerate(axes[1][1]):
                iy = (ix + (axes[1][0] + k).remainder(dims)) * dims
                wxy = wx * wy if m is None else wx * wy * m
                for q, wz in enumerate(axes[2][1]):
                    grid.index_add_(0, iy + (axes[2][0] + q).remainder(dims), wxy * wz)
    return grid.reshape(dims, dims, dims)


def _window(dims, p):
    """(x / sin x)^p of every FFT index, x = pi k / dims."""
    k = torch.arange(dims, device=_device(), dtype=torch.float64)
    k = torch.where(k > dims // 2, k - dims, k)
    x = math.pi * k / dims
    return k, torch.where(k == 0, torch.ones_like(x), (x / torch.sin(x)) ** p)


class _Modes(object):
    """The independent modes of a real field: wave numbers, bins and line of sight."""

    def __init__(self, dims, axis):
        k, _ = _window(dims, 0)
        k = k.long()
        nz, mid = dims // 2 + 1, dims // 2
        kx, ky, kz = k[:, None, None], k[None, :, None], torch.arange(nz, device=_device())[None, None, :]
        edge = (kz == 0) | ((kz == mid) & (dims % 2 == 0))
        edge_x = (kx == 0) | ((kx == mid) & (dims % 2 == 0))
        self.dims = dims
        self.keep = ~(edge & ((kx < 0) | (edge_x & (ky < 0))))
        n2 = kx * kx + ky * ky + kz * kz
        par = (kx, ky, kz)[axis].expand_as(n2)
        self.n2 = n2[self.keep]
        self.par = par[self.keep].abs()
        self.mu2 = torch.where(self.n2 > 0, self.par.double() ** 2 / self.n2.clamp_min(1).double(), 0.0)
        self.bin3 = torch.floor(torch.sqrt(self.n2.double())).long()
        per = torch.floor(torch.sqrt((self.n2 - self.par ** 2).double())).long()
        self.inside = self.n2 <= mid * mid
        self.nb1, self.nper = mid + 1, int(math.sqrt(2.0 * mid * mid)) + 1
        self.nb3 = int(math.sqrt(3.0 * mid * mid)) + 1
        self.bin2 = (mid + 1) * per + self.par

    def sums(self, v, which):
        if which == 3:
            return torch.bincount(self.bin3, v, self.nb3)
        if which == 2:
            return torch.bincount(self.bin2, v, self.nb1 * self.nper)
        return torch.bincount(self.par[self.inside], v[self.inside], self.nb1)

    def legendre(self):
        m = self.mu2
        return [torch.ones_like(m), 0.5 * (3.0 * m - 1.0), 0.125 * ((35.0 * m - 30.0) * m + 3.0)]


def _transform(grid, other, p):
    """The float64 half-complex field, interlaced with `other`, the window divided out."""
    dims = grid.shape[0]
    d = torch.fft.rfftn(grid.double())
    k, win = _window(dims, p)
    kz, wz = torch.arange(dims // 2 + 1, device=_device(), dtype=torch.float64), win[:dims // 2 + 1]
    if other is not None:
        phase = (k[:, None, None] + k[None, :, None] + kz[None, None, :]) * (math.pi / dims)
        d = 0.5 * (d + torch.fft.rfftn(other.double()) * torch.polar(torch.ones_like(phase), phase))
    return d * (win[:, None, None] * win[None, :, None] * wz[None, None, :])


def _auto_sums(grid, other, mas, axis):
    m = _Modes(grid.shape[0], axis)
    d = _transform(grid, other, SUPPORT[mas])[m.keep]
    p = d.real ** 2 + d.imag ** 2
    phase = torch.atan2(d.real, torch.sqrt(p))
    return (m, [m.sums(p * l, 3) for l in m.legendre()], m.sums(phase * phase, 3), m.sums(p, 1), m.sums(p, 2))


def _geometry(m):
    """Mean wave numbers and mode counts of the 1D and 3D bins, centres of the 2D bins."""
    kf = 2.0 * math.pi / BOX
    one = torch.ones_like(m.mu2)
    n1, n2, n3 = (m.sums(one, j) for j in (1, 2, 3))
    k1 = kf * torch.arange(m.nb1, device=_device(), dtype=torch.float64)[1:]
    k3 = kf * (m.sums(torch.sqrt(m.n2.double()), 3) / n3)[1:]
    i = torch.arange(m.nb1 * m.nper, device=_device())
    cells = dict(kpar=((i % m.nb1).double() + 0.5) * kf, kper=((i // m.nb1).double() + 0.5) * kf)
    area = math.pi * (((m.nb1 - 1) * kf) ** 2 - k1 ** 2) / n1[1:] / (2.0 * math.pi) ** 2
    return n1, n2, n3, area, dict(k1D=k1, k3D=k3, Nmodes1D=n1[1:], Nmodes2D=n2, Nmodes3D=n3[1:], **cells)


def _finish(m, p3, ph, p1, p2):
    f = (BOX / m.dims ** 2) ** 3
    n1, n2, n3, area, out = _geometry(m)
    out.update(Pk=torch.stack([c * x[1:] / n3[1:] * f for c, x in zip((1.0, 5.0, 9.0), p3)], 1),
               Pkphase=ph[1:] / n3[1:] * f, Pk1D=p1[1:] * f * area, Pk2D=p2 * f / n2)
    return {k: v.cpu().numpy() for k, v in out.items()}


def _exact_auto(grid, other, mas, axis):
    return _finish(*_auto_sums(grid, other, mas, axis))


def _exact_cross(fields, schemes, axis):
    dims = fields[0].shape[0]
    m, f = _Modes(dims, axis), (BOX / dims ** 2) ** 3
    ds = [_transform(x, None, SUPPORT[s])[m.keep] for x, s in zip(fields, schemes)]
    n = len(ds)
    n1, n2, n3, area, out = _geometry(m)
    legendre = m.legendre()

    def spectra(pairs):
        a, b, c = [], [], []
        for i, j in pairs:
            v = ds[i].real * ds[j].real + ds[i].imag * ds[j].imag
            a.append(torch.stack([q * m.sums(v * l, 3)[1:] / n3[1:] * f for q, l in zip((1.0, 5.0, 9.0), legendre)], 1))
            b.append(m.sums(v, 1)[1:] * f * area)
            c.append(m.sums(v, 2) * f / n2)
        return [torch.stack(x, -1) for x in (a, b, c)]

    out['Pk'], out['Pk1D'], out['Pk2D'] = spectra([(i, i) for i in range(n)])
    out['XPk'], out['PkX1D'], out['PkX2D'] = spectra([(i, j) for i in range(n) for j in range(i + 1, n)])
    return {k: v.cpu().numpy() for k, v in out.items()}


def _exact_xi(delta, mas, axis):
    dims = delta.shape[0]
    d = _transform(delta, None, SUPPORT[mas])
    xi = torch.fft.irfftn(d.real ** 2 + d.imag ** 2, s=(dims,) * 3).reshape(-1)
    k, _ = _window(dims, 0)
    r = k.long()
    r2 = r[:, None, None] ** 2 + r[None, :, None] ** 2 + r[None, None, :] ** 2
    par = r.reshape([-1 if a == axis else 1 for a in range(3)]).expand_as(r2).reshape(-1)
    r2 = r2.reshape(-1)
    mu2 = torch.where(r2 > 0, par.double() ** 2 / r2.clamp_min(1).double(), 0.0)
    length = torch.sqrt(r2.double())
    b = torch.floor(length).long()
    nb = int(math.sqrt(3.0 * (dims // 2) ** 2)) + 1
    n = torch.bincount(b, minlength=nb).double()
    terms = (1.0, 2.5 * (3.0 * mu2 - 1.0), 1.125 * ((35.0 * mu2 - 30.0) * mu2 + 3.0))
    mult = torch.stack([torch.bincount(b, xi * t, nb)[1:] / n[1:] for t in terms], 1) / float(dims) ** 3
    return dict(r3D=(torch.bincount(b, length, nb) / n)[1:].cpu().numpy() * (BOX / dims),
                Nmodes3D=n[1:].cpu().numpy(), xi=mult.cpu().numpy())


def _exact_bk(case, delta):
    dims = delta.shape[0]
    k1, k2, theta = _triangles(case)
    k3 = np.sqrt((k2 * np.sin(theta)) ** 2 + (k2 * np.cos(theta) + k1) ** 2)
    kf = 2.0 * math.pi / BOX
    d = _transform(delta, None, SUPPORT[case['mas']])
    k, _ = _window(dims, 0)
    kz = torch.arange(dims // 2 + 1, device=_device(), dtype=torch.float64)
    kk = torch.sqrt(k[:, None, None] ** 2 + k[None, :, None] ** 2 + kz[None, None, :] ** 2)

    def shell(q):
        inside = ((kk >= (q - kf) / kf) & (kk < (q + kf) / kf)).double()
        x, one = torch.fft.irfftn(d * inside, s=(dims,) * 3), torch.fft.irfftn(inside + 0j, s=(dims,) * 3)
        return x, one, float((x * x).sum() / (one * one).sum()) * (BOX / dims ** 2) ** 3

    a, ia, pa = shell(k1)
    b, ib, pb = shell(k2)
    a, ia = a * b, ia * ib
    bs, qs, ps = [], [], []
    for q in k3:
        c, ic, pc = shell(float(q))
        bs.append(float((a * c).sum() / (ia * ic).sum()) * (BOX ** 2 / dims ** 3) ** 3)
        qs.append(bs[-1] / (pa * pb + pa * pc + pb * pc))
        ps.append(pc)
    return dict(B=np.array(bs), Q=np.array(qs), k=np.concatenate([[k1, k2], k3]), Pk=np.array([pa, pb] + ps))


def _adds(case):
    if case['kind'] == 'batch':
        return sum(_adds(dict(kind='chain', dims=s['dims'], n=s['n'], mas=s['MAS'], interlaced=s['interlaced']))
                   for s in _specs(case))
    n = case.get('n') or case['side'] ** 3
    return n * SUPPORT[case['mas']] ** 3 * (2 if case['interlaced'] else 1)


def _overdensities(pos, dims, mas, interlaced):
    shifts = (0.0, 0.5) if interlaced else (0.0,)
    out = [_deposit(pos, None, dims, mas, s) * (float(dims) ** 3 / pos.shape[0]) - 1.0 for s in shifts]
    return out[0], out[1] if interlaced else None


def exact(case, seed):
    kind = case['kind']
    if kind in ('ma', 'chain', 'batch') and _adds(case) > EXACT_ADDS:
        return None
    if kind == 'chain' and case['dims'] > 640:
        return None
    g = _generator(seed)
    if kind == 'batch':
        out = []
        for s in _specs(case):
            pos = torch.rand((s['n'], 3), generator=g, device=_device()) * (BOX * (1 - 1e-6))
            grid, other = _overdensities(pos, s['dims'], s['MAS'], s['interlaced'])
            _, p3, ph, p1, p2 = _auto_sums(grid, other, s['MAS'], case['axis'])
            out.append(torch.cat([torch.stack(p3, 1).reshape(-1), ph, p1, p2]))
        return out
    if kind == 'chain':
        pos = _particles(case['side'], g, case['order'])
        grid, other = _overdensities(pos, case['dims'], case['mas'], case['interlaced'])
        return _exact_auto(grid, other, case['mas'], case['axis'])
    state = prepare(case, seed)
    if kind == 'ma':
        pos, w = state['pos'], state['w']
        if case['host']:
            pos = torch.from_numpy(pos).to(_device())
            w = None if w is None else torch.from_numpy(w).to(_device())
            return _deposit(pos, w, case['dims'], case['mas'], 0.0).cpu().numpy()
        return [_deposit(pos, w, case['dims'], case['mas'], s) for s in ((0.0, 0.5) if case['interlaced'] else (0.0,))]
    if kind == 'interp':
        x, f, d = state['pos'].double() * (case['dims'] / BOX), state['field'].double().reshape(-1), case['dims']
        axes = [_weights(x[:, a], 'CIC') for a in range(3)]
        den = torch.zeros(x.shape[0], dtype=torch.float64, device=_device())
        for c in range(8):
            bits = (c >> 2, (c >> 1) & 1, c & 1)
            ix, iy, iz = ((axes[a][0] + bits[a]).remainder(d) for a in range(3))
            den += f[(ix * d + iy) * d + iz] * axes[0][1][bits[0]] * axes[1][1][bits[1]] * axes[2][1][bits[2]]
        return den
    if kind == 'pk':
        return _exact_auto(state['delta'], state['other'], case['mas'], case['axis'])
    if kind == 'xpk':
        return _exact_cross(state['fields'], _schemes(case), case['axis'])
    if kind == 'xi':
        return _exact_xi(state['delta'], case['mas'], case['axis'])
    return _exact_bk(case, state['delta'])
