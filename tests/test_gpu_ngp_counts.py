"""Unweighted NGP of a million particles and more on grids in L2 (whole-number counts)
against exact counts: lattice and random order, runs in one cell, positions outside the box
and not finite, one and two grids, onto a filled grid; the tiled deposit gives the same
bits, also where the workspace is too small for the counts."""
import numpy as np
import pytest
import torch

import oracle as O

pytestmark = pytest.mark.gpu
BOX = 1000.0


@pytest.mark.parametrize('inter', [False, True])
@pytest.mark.parametrize('dims,n', [(7, 2 ** 20), (64, 2 ** 20 + 33), (129, 2 ** 20 + 1), (203, 3000001), (256, 2 ** 21)])
def test_counts(dims, n, inter):
    import pylians_gb300.build as b
    b.build()
    import pylians_gb300.MAS_library as MASL
    from pylians_gb300 import _lib
    from pylians_gb300._device import ptr, stream_ptr
    r = np.random.default_rng(dims)
    pos = (r.random((n, 3)) * BOX).astype(np.float32)
    pos[: n // 3] = pos[: n // 3][np.argsort(pos[: n // 3, 0])]
    pos[n // 2: n // 2 + 5000] = pos[n // 2]                 # a run in one cell
    pos[:3] = [[BOX, 0.0, -1.0], [-0.5 * BOX / dims, 2.3 * BOX, 5.0], [np.nextafter(np.float32(BOX), 0)] * 3]
    base = r.integers(0, 9, (dims,) * 3).astype(np.float32)
    dev = torch.from_numpy(pos).cuda()

    def run(strategy):
        g = [torch.from_numpy(base.copy()).cuda() for _ in range(2)]
        MASL.MA(dev, g[0], BOX, 'NGP', interlaced=g[1] if inter else None, strategy=strategy)
        return [x.cpu().numpy() for x in g]
    got, tiled = run('auto'), run('tiled')
    for k in range(1 + inter):
        ref = base.astype(np.float64)
        O.ma_acc64((pos + np.float32(0.5 * BOX / dims)).astype(np.float32) if k else pos, ref, BOX, 'NGP')
        assert np.array_equal(got[k], ref) and np.array_equal(got[k], tiled[k])
    # not finite: the same cells as the tiled deposit
    dev[5:8] = torch.tensor([[float('nan')] * 3, [float('inf'), 1.0, 2.0], [1.0, -float('inf'), 1e30]], device='cuda')
    assert all(np.array_equal(x, y) for x, y in zip(run('auto'), run('tiled')))
    # a workspace for the tiled deposit alone
    L = _lib.load()
    small = L.pyl_ma_workspace_size(n, 3, dims, 1, 2, int(inter))
    g = [torch.from_numpy(base.copy()).cuda() for _ in range(2)]
    ws = torch.empty(small, dtype=torch.uint8, device='cuda')
    _lib.call('pyl_ma', ptr(dev), None, n, 3, ptr(g[0]), ptr(g[1]) if inter else None, dims, BOX, 1, 0, 1, ptr(ws), small,
              stream_ptr())
    assert all(np.array_equal(x.cpu().numpy(), y) for x, y in zip(g, run('tiled')))
