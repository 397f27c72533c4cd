"""Deposits whose bins go to several CTAs in parts (few bins, many particles), tiled and
batched, against float64 sums of the oracle's weights: even particles and a box that holds
half of them (the last part of its bins takes what the others leave, and some of its
cells pass 512, whose parts are summed in float32), grids of one bin and of a few, sides
that are no multiple of a bin, weights in fixed point and in float32.

Tolerance: a cell holds at most some 2^10 particles, 2^13 contributions or fewer, each
exact to 2^-23 (of the largest weight) in fixed point; a float32 sum of them is off by
at most half an ulp of the cell each, 2^6 ulps with independent roundings, and the
halos of up to 8 bins are added in float32: 2^7 * 2^-24 of the largest cell, and 2^13 *
2^-23 of the largest weight.  NGP counts are exact."""
import numpy as np
import pytest
import torch

import oracle as O

pytestmark = pytest.mark.gpu
BOX = 1000.0


@pytest.fixture(scope='module')
def mods():
    import pylians_gb300.build as b
    b.build()
    import pylians_gb300.MAS_library as MASL
    from pylians_gb300 import batch
    return MASL, batch


def particles(n, crowded, seed):
    r = np.random.default_rng(seed)
    pos = r.random((n, 3))
    if crowded:
        pos[: n // 2] = 0.2 + 0.3 * pos[: n // 2]
    pos = (pos * BOX).astype(np.float32)
    pos[pos >= BOX] = 0.0
    return pos


def reference(pos, dims, mas, shift, w=None):
    g = np.zeros((dims,) * 3)
    p = (pos + np.float32(0.5 * BOX / dims)).astype(np.float32) if shift else pos
    O.ma_acc64(p, g, BOX, mas, w)
    return g


def check(got, ref, wmax=1.0):
    assert np.abs(got - ref).max() <= 2.0 ** -17 * np.abs(ref).max() + 2.0 ** -10 * wmax


@pytest.mark.parametrize('crowded', [False, True])
@pytest.mark.parametrize('dims,mas,inter,weights', [
    (16, 'CIC', True, None), (32, 'NGP', False, None), (33, 'TSC', False, 'narrow'), (64, 'PCS', True, None),
    (64, 'NGP', True, 'narrow'), (80, 'PCS', False, 'wide'), (128, 'PCS', True, None), (70, 'CIC', False, None)])
def test_tiled_parts(mods, dims, mas, inter, weights, crowded):
    MASL, _ = mods
    bins = (-(-dims // 32)) ** 3
    s = {'NGP': 1, 'CIC': 2, 'TSC': 3, 'PCS': 4}[mas]
    n = int(2.5 * bins * 2 ** 20 / (s ** 3 * (2 if inter else 1)))       # two and a half parts a bin
    pos, w = particles(n, crowded, dims), None
    if weights:
        w = np.exp(np.random.default_rng(1).standard_normal(n) * (0.1 if weights == 'narrow' else 2.0)).astype(np.float32)
    g = torch.zeros((2 if inter else 1,) + (dims,) * 3, device='cuda')
    MASL.MA(torch.from_numpy(pos).cuda(), g[0], BOX, mas, None if w is None else torch.from_numpy(w).cuda(),
            interlaced=g[1] if inter else None, strategy='tiled')
    for k in range(2 if inter else 1):
        ref, got = reference(pos, dims, mas, k, w), g[k].cpu().numpy()
        if mas == 'NGP' and w is None:
            assert np.array_equal(got, ref)
        check(got, ref, 1.0 if w is None else w.max())


def test_batched_parts(mods):
    _, batch = mods
    specs = [dict(dims=64, MAS='PCS', interlaced=True, n=400001), dict(dims=32, MAS='TSC', interlaced=False, n=90000),
             dict(dims=64, MAS='CIC', interlaced=False, n=70), dict(dims=32, MAS='NGP', interlaced=True, n=2200000),
             dict(dims=40, MAS='CIC', interlaced=True, n=1300000), dict(dims=96, MAS='TSC', interlaced=False, n=5)]
    pos = [particles(s['n'], i % 2 == 0, i) for i, s in enumerate(specs)]
    b = batch.RealizationBatch(specs, BOX, tune=False, method='tiled')
    b.step([torch.from_numpy(p).cuda() for p in pos])
    for s, p in zip(b.specs, pos):
        scale = s['dims'] ** 3 / s['n']
        for k in range(2 if s['interlaced'] else 1):
            got = b.grids[s['dims']][s['slot2'] if k else s['slot']].cpu().numpy()
            ref = reference(p, s['dims'], s['MAS'], k) * scale - 1.0
            check(got, ref, scale)


@pytest.mark.parametrize('offset', [2.0 ** -5, 2.0 ** -6])
@pytest.mark.parametrize('mas', ['TSC', 'PCS'])
def test_small_cells_beside_crowded_ones(mas, offset):
    """2^18 particles at one point of 64^3 (cells of unit length, so every weight follows
    from `offset` alone): each part of the bin is redone in float32 for its cells past 512,
    and the cells of the smallest weights, far below 2^-22, keep float32's relative error,
    at most one rounding of 2^-24 for each addition and eight for a weight."""
    import pylians_gb300.build as b
    b.build()
    import pylians_gb300.MAS_library as MASL
    n, dims = 1 << 18, 64
    o = {'TSC': 0.5, 'PCS': 0.0}[mas] + 1.0 - offset
    pos = torch.tensor([20.0 + o, 20.0 + o, 20.25], device='cuda').expand(n, 3).contiguous()
    grid = torch.zeros((dims,) * 3, device='cuda')
    MASL.MA(pos, grid, float(dims), mas, strategy='tiled')
    ref = torch.zeros((dims,) * 3, dtype=torch.float64, device='cuda')
    near = [], [], []
    for a in range(3):
        x = float(pos[0, a])
        for k in range(int(x) - 3, int(x) + 5):
            s = abs(x - k)
            if mas == 'TSC':
                w = 0.75 - s * s if s < 0.5 else 0.5 * max(1.5 - s, 0.0) ** 2
            else:
                w = (4 - 6 * s * s + 3 * s ** 3) / 6 if s < 1 else max(2 - s, 0.0) ** 3 / 6
            near[a].append((k, w))
    for i, wi in near[0]:
        for j, wj in near[1]:
            for k, wk in near[2]:
                ref[i, j, k] = n * wi * wj * wk
    assert bool(((grid.double() - ref).abs() <= (n + 24) * 2.0 ** -24 * ref).all())


@pytest.mark.parametrize('interlaced', [False, True])
def test_batch_of_more_particles_than_the_stated_total(mods, interlaced):
    """A stated total below the items' particles keeps that many records, in bins whose
    parts then have no shared words: whole bins.  A particle's weights add up to 1 within
    27 units of 2^-22."""
    from pylians_gb300 import _lib
    from pylians_gb300._device import ptr, stream_ptr
    _, batch = mods
    n, total, dims = 400000, 1000, 32
    g = torch.Generator(device='cuda')
    g.manual_seed(5)
    pos = torch.rand((n, 3), generator=g, device='cuda') * (BOX * 0.99)
    b = batch.RealizationBatch([dict(dims=dims, MAS='TSC', interlaced=interlaced, n=n)], BOX, tune=False, method='tiled')
    b._tables([pos])
    b.grids[dims].zero_()
    nbytes = _lib.load().pyl_ma_batch_tiled_workspace_size(b.total_tiles, total)
    ws = torch.full((nbytes,), 255, dtype=torch.uint8, device='cuda')
    _lib.call('pyl_ma_batch_tiled', ptr(b.reals_dev), 1, ptr(b.items_dev), b.n_items, ptr(b.tile_base), b.total_tiles,
              total, ptr(ws), nbytes, 4, stream_ptr())
    scale = dims ** 3 / n
    for k in range(2 if interlaced else 1):
        got = float(b.grids[dims][b.specs[0]['slot2'] if k else b.specs[0]['slot']].double().sum())
        assert abs(got - total * scale) <= total * scale * 32 * 2.0 ** -22


def test_crowded_cells_of_parts_cost_little(mods):
    """2^22 particles on 64^3, a twentieth of them in 50 clumps of 1 Mpc/h (2.5 times the
    uniform time where each addition to a crowded cell returns its old value)."""
    MASL, _ = mods
    n, dims = 1 << 22, 64
    g = torch.Generator(device='cuda')
    g.manual_seed(1)
    u = torch.rand((n, 3), generator=g, device='cuda') * (BOX * 0.999)
    c = u.clone()
    m = n // 20
    c[:m] = (u[:50][torch.randint(50, (m,), generator=g, device='cuda')] +
             torch.randn((m, 3), generator=g, device='cuda')).clamp(0.0, BOX * 0.999)
    c = c[torch.randperm(n, generator=g, device='cuda')].contiguous()
    grid, best = torch.zeros((dims,) * 3, device='cuda'), []
    for p in (u, c):
        times = []
        for _ in range(5):
            t0, t1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            t0.record()
            MASL.MA(p, grid, BOX, 'CIC')
            t1.record()
            torch.cuda.synchronize()
            times.append(t0.elapsed_time(t1))
        best.append(min(times[1:]))
    assert best[1] <= 1.6 * best[0]


@pytest.mark.parametrize('dims,mas,inter,parts', [(128, 2, 1, 16), (64, 2, 0, 8), (64, 4, 1, 128)])
def test_average_bins_of_less_than_two_parts_stay_whole(mods, dims, mas, inter, parts):
    """The workspace has room for the grids' words only from two parts (of 2^20 additions,
    `parts` a particle) an average bin on."""
    from pylians_gb300 import _lib
    size = _lib.load().pyl_ma_workspace_size
    bins, n = (dims // 32) ** 3, 2 * (dims // 32) ** 3 * (1 << 20) // parts
    words = 8 * dims ** 3 * (2 if inter else 1)
    assert size(n, 3, dims, mas, 2, inter) - size(n - bins, 3, dims, mas, 2, inter) >= words
    assert size(n - bins, 3, dims, mas, 2, inter) - size(n - 2 * bins, 3, dims, mas, 2, inter) < words // 4


@pytest.mark.parametrize('dims', [64, 114])
@pytest.mark.parametrize('mas,inter', [('CIC', 0), ('TSC', 1), ('PCS', 0)])
def test_parts_round_cells_as_whole_bins_do(mods, dims, mas, inter):
    """The same deposit with a workspace that has no room for the words (whole bins): the
    same bits in every cell that one or two bins add to (three and more meet in any order)."""
    from pylians_gb300 import _lib
    from pylians_gb300._device import ptr, stream_ptr
    s = {'CIC': 2, 'TSC': 3, 'PCS': 4}[mas]
    bins = (-(-dims // 32)) ** 3
    n = int(3 * bins * (1 << 20) / (s ** 3 * (1 + inter)))
    g = torch.Generator(device='cuda')
    g.manual_seed(dims)
    pos = torch.rand((n, 3), generator=g, device='cuda') * (BOX * 0.999)
    size = _lib.load().pyl_ma_workspace_size(n, 3, dims, s, 2, inter)
    words = 8 * bins * (32 + s - 1 + inter) ** 3 * (1 + inter)
    out = []
    for nbytes in (size, size - words):
        ws = torch.empty(nbytes, dtype=torch.uint8, device='cuda')
        grids = torch.zeros((1 + inter, dims, dims, dims), device='cuda')
        _lib.call('pyl_ma', ptr(pos), None, n, 3, ptr(grids[0]), ptr(grids[1]) if inter else None, dims, BOX, s, 2, 0, ptr(ws),
                  nbytes, stream_ptr())
        out.append(grids.cpu().numpy())
    k = np.arange(dims)
    halo = k % 32 < s - 1 + inter
    if dims % 32:                            # the last bin is cut off: its halo wraps onto more
        halo |= k % 32 < (s - 1 + inter + 32 - dims % 32)
    h = halo[:, None, None].astype(int) + halo[None, :, None] + halo[None, None, :]
    cells = h <= 1
    assert cells.mean() > 0.3
    for i in range(1 + inter):
        assert np.array_equal(out[0][i][cells], out[1][i][cells])
