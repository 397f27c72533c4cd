"""The record sort of the deterministic strategy with one to four 8-bit passes (grids of up
to 2^8, 2^16, 2^24 and more cells), tiles of 4096 records that end inside, at and after the
last one, with and without weights: NGP counts are exact and weights that are small whole
numbers add exactly, so that a lost, doubled or misplaced particle shows; TSC against
float64 sums, a cell's float32 sum of at most 2^10 products within 2^10 * 2^-24 of it."""
import numpy as np
import pytest
import torch

import oracle as O

pytestmark = pytest.mark.gpu
BOX = 1000.0


@pytest.mark.parametrize('weighted', [False, True])
@pytest.mark.parametrize('dims,n', [(6, 100), (7, 4095), (40, 4096), (41, 4097), (256, 100000), (257, 3 * 4096 + 1)])
def test_passes(dims, n, weighted):
    import pylians_gb300.build as b
    b.build()
    import pylians_gb300.MAS_library as MASL
    r = np.random.default_rng(n)
    pos = (r.random((n, 3)) * BOX).astype(np.float32)
    pos[pos >= BOX] = 0.0
    w = r.integers(1, 8, n).astype(np.float32) if weighted else None
    dev = [torch.from_numpy(x).cuda() if x is not None else None for x in (pos, w)]
    for mas in ('NGP', 'TSC'):
        g = [torch.zeros((dims,) * 3, device='cuda') for _ in range(2)]
        MASL.MA(dev[0], g[0], BOX, mas, dev[1], interlaced=g[1], strategy='sorted')
        for k in range(2):
            ref = np.zeros((dims,) * 3)
            O.ma_acc64((pos + np.float32(0.5 * BOX / dims)).astype(np.float32) if k else pos, ref, BOX, mas, w)
            got = g[k].cpu().numpy()
            if mas == 'NGP':
                assert np.array_equal(got, ref)
            else:
                assert (np.abs(got - ref) <= 2.0 ** -14 * ref).all()
