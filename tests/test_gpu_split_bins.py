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
