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


@pytest.mark.parametrize('inter', [False, True])
@pytest.mark.parametrize('points', [1, 2, 3, 16, 33, 64])
def test_few_cells_in_no_order(points, inter):
    """All particles at a few points, in no order: exact counts, the last warp part empty."""
    import pylians_gb300.build as b
    b.build()
    import pylians_gb300.MAS_library as MASL
    n, dims = (1 << 20) + 5, 64
    g = torch.Generator(device='cuda')
    g.manual_seed(points)
    cells = torch.randperm(dims ** 3, generator=g, device='cuda')[:points]
    k = cells[torch.randint(points, (n,), generator=g, device='cuda')]
    pos = torch.stack([k // dims ** 2, k // dims % dims, k % dims], 1).float() + 0.25
    grids = [torch.zeros((dims,) * 3, device='cuda') for _ in range(2 if inter else 1)]
    MASL.MA(pos, grids[0], float(dims), 'NGP', interlaced=grids[1] if inter else None)
    for s, grid in zip((0.0, 0.5), grids):
        c = (pos + (s + 0.5)).floor().long() % dims
        ref = torch.bincount((c[:, 0] * dims + c[:, 1]) * dims + c[:, 2], minlength=dims ** 3)
        assert bool((grid.reshape(-1) == ref).all())


def test_few_cells_in_no_order_cost_little():
    """2^24 particles at 4 points of 128^3: additions queue in four words (30 times the
    time of as many all over the box, each added by itself)."""
    import pylians_gb300.build as b
    b.build()
    import pylians_gb300.MAS_library as MASL
    n, dims = 1 << 24, 128
    g = torch.Generator(device='cuda')
    g.manual_seed(1)
    u = torch.rand((n, 3), generator=g, device='cuda') * (dims - 0.01)
    few = u[:4][torch.randint(4, (n,), generator=g, device='cuda')].contiguous()
    grid, best = torch.zeros((dims,) * 3, device='cuda'), []
    for p in (u, few):
        times = []
        for _ in range(4):
            t0, t1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            t0.record()
            MASL.MA(p, grid, float(dims), 'NGP')
            t1.record()
            torch.cuda.synchronize()
            times.append(t0.elapsed_time(t1))
        best.append(min(times[1:]))
    assert best[1] <= 12.0 * best[0]
