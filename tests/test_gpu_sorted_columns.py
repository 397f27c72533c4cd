"""The deterministic strategy's column deposit against float64 sums of the oracle's
weights: grids smaller than the support of a particle, sides at the edges of its CTAs
(14 to 16 columns of x, 29 to 32 of y, 32 layers of z), empty and crowded columns, with
and without weights and interlacing, onto a filled grid.

Tolerance: a cell's float32 sum of m contributions is off by at most m ulps; with
independent roundings sqrt(m), m below 2^16 in the crowded cells: 2^8 * 2^-24 of the
largest cell.  Unweighted NGP counts are exact, and two runs give the same bits."""
import numpy as np
import pytest
import torch

import oracle as O

pytestmark = pytest.mark.gpu
BOX = 1000.0


@pytest.mark.parametrize('mas', ['NGP', 'CIC', 'TSC', 'PCS'])
@pytest.mark.parametrize('dims,n', [(1, 300), (2, 300), (3, 5), (13, 4000), (14, 1), (16, 20000), (29, 9000),
                                    (31, 50000), (33, 20000), (65, 3000), (96, 400000)])
def test_columns_equal_float64(mas, dims, n):
    import pylians_gb300.build as b
    b.build()
    import pylians_gb300.MAS_library as MASL
    r = np.random.default_rng(dims)
    pos = r.random((n, 3))
    pos[: n // 4] = 0.5 + 0.02 * pos[: n // 4]              # a crowded spot
    pos = (pos * BOX).astype(np.float32)
    pos[pos >= BOX] = 0.0
    w = r.lognormal(size=n).astype(np.float32) if dims % 2 else None
    base = r.random((dims,) * 3).astype(np.float32)
    if w is None:
        base = np.round(base)
    out = []
    for _ in range(2):
        g = [torch.from_numpy(base.copy()).cuda() for _ in range(2)]
        MASL.MA(torch.from_numpy(pos).cuda(), g[0], BOX, mas, None if w is None else torch.from_numpy(w).cuda(),
                interlaced=g[1], strategy='sorted')
        out.append([x.cpu().numpy() for x in g])
    for k in range(2):
        ref = base.astype(np.float64)
        O.ma_acc64((pos + np.float32(0.5 * BOX / dims)).astype(np.float32) if k else pos, ref, BOX, mas, w)
        assert np.array_equal(out[0][k], out[1][k])
        assert np.abs(out[0][k] - ref).max() <= 256 * 2.0 ** -24 * np.abs(ref).max()
        if mas == 'NGP' and w is None:
            assert np.array_equal(out[0][k], ref)
