"""Batched placement with one bin to 4096 bins per realization (more than one per thread of
its scan, and more than its threads) and particle counts around its batches of 2048: NGP
counts are exact, so that a lost or misplaced particle shows."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize('dims', [20, 33, 257, 270, 512])
def test_ngp_counts(dims):
    import pylians_gb300.build as b
    b.build()
    from pylians_gb300 import batch
    box = float(dims)
    specs = [dict(dims=dims, MAS='NGP', interlaced=False, n=n) for n in (1, 2047, 2048, 2049, 100003)]
    r = np.random.default_rng(dims)
    pos = [(r.random((s['n'], 3)) * box).astype(np.float32) for s in specs]
    B = batch.RealizationBatch(specs, box, axis=0, method='tiled', tune=False)
    B.step([torch.from_numpy(p).cuda() for p in pos])
    for i, (s, p) in enumerate(zip(specs, pos)):
        cell = np.floor(p.astype(np.float64) + 0.5).astype(np.int64) % dims
        ref = np.bincount((cell[:, 0] * dims + cell[:, 1]) * dims + cell[:, 2], minlength=dims ** 3)
        got = (B.grids[dims][i].cpu().numpy().astype(np.float64).ravel() + 1.0) * s['n'] / dims ** 3
        # overdensity = count * dims^3 / n - 1 in float32: one rounding of the product, one of the sum
        assert np.abs(got - ref).max() <= 2.0 ** -23 * max(1.0, ref.max())


def test_few_large_items_are_divided():
    """Two realizations of 3 million particles in items of 65536 (92 of them) take little
    more than in items of 4096 (1.6 times with an item to a CTA), and give the same counts."""
    import pylians_gb300.build as b
    b.build()
    from pylians_gb300 import batch
    dims, n = 128, 3000000
    g = torch.Generator(device='cuda')
    g.manual_seed(1)
    pos = [torch.rand((n, 3), generator=g, device='cuda') * (dims - 0.01) for _ in range(2)]
    times, grids = [], []
    for item in (4096, 65536):
        B = batch.RealizationBatch([dict(dims=dims, MAS='NGP', interlaced=False, n=n)] * 2, float(dims), method='tiled',
                                   tune=False)
        B.item_sizes = [item] * 2
        t = []
        for _ in range(5):
            t0, t1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            t0.record()
            for _ in range(4):
                B.step(pos)
            t1.record()
            torch.cuda.synchronize()
            t.append(t0.elapsed_time(t1))
        times.append(min(t))
        grids.append(B.grids[dims].clone())
    assert torch.equal(*grids)
    assert times[1] <= 1.25 * times[0]
