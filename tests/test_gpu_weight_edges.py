"""TSC and PCS weights at the edges of their formulas: coordinates at, and one float32
step to either side of, cell edges and half cells, and coordinates far outside the box,
below and above the 2^22 cells up to which each weight has one formula.

Tolerance: one particle per 8^3 cells, so that a cell holds one product of three weights;
each weight is off from the oracle's double arithmetic by at most 2^-22 (roundings of
numbers below 8, over six), the fixed-point sum by another 2^-22: 2^-20 together."""
import numpy as np
import pytest
import torch

import oracle as O

pytestmark = pytest.mark.gpu
N = 64


@pytest.mark.parametrize('strategy', ['atomic', 'tiled', 'sorted'])
@pytest.mark.parametrize('mas', ['TSC', 'PCS'])
@pytest.mark.parametrize('shift', [0, -128, 2 ** 22 - 64, 2 ** 22, 2 ** 23])
def test_weight_edges(mas, shift, strategy):
    import pylians_gb300.build as b
    b.build()
    import pylians_gb300.MAS_library as MASL
    r = np.random.default_rng(5)
    cells = np.stack(np.meshgrid(*[np.arange(0, N, 8)] * 3, indexing='ij'), -1).reshape(-1, 3)
    edges = np.array([0.0, 2.0 ** -30, 0.25, 0.5, 0.75, 1.0 - 2.0 ** -20])
    x = (cells + shift + edges[r.integers(0, len(edges), cells.shape)]).astype(np.float32)
    x = np.nextafter(x, (x + r.integers(-1, 2, x.shape)).astype(np.float32)).astype(np.float32)
    ref = np.zeros((N,) * 3)
    O.ma_acc64(x, ref, float(N), mas, None)
    g = torch.zeros((N,) * 3, device='cuda')
    MASL.MA(torch.from_numpy(x).cuda(), g, float(N), mas, strategy=strategy)
    assert np.abs(g.cpu().numpy() - ref).max() <= 2.0 ** -20
