"""The sorted strategy on particles that leave most of the box empty or crowd a few cells:
float64 sums of the grids, and times in proportion to those of a uniform box, so that no
thread is left with work that grows with the empty part or the crowded one.

The bounds on times lie well below what one thread doing such work takes (in brackets)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

BOX = 1000.0


@pytest.fixture(scope='module')
def MASL():
    import pylians_gb300.build as b
    b.build()
    import pylians_gb300.MAS_library as MASL
    return MASL


def uniform(n, seed=1, part=1.0):
    g = torch.Generator(device='cuda')
    g.manual_seed(seed)
    return torch.rand((n, 3), generator=g, device='cuda') * (BOX * part * (1 - 1e-6))


def time_us(MASL, pos, dims, mas, w=None):
    grid = torch.zeros((dims,) * 3, device='cuda')
    times = []
    for _ in range(4):
        t0, t1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        t0.record()
        MASL.MA(pos, grid, BOX, mas, w, strategy='sorted')
        t1.record()
        torch.cuda.synchronize()
        times.append(t0.elapsed_time(t1) * 1e3)
    return min(times[1:])


def test_empty_part_of_the_box_costs_nothing(MASL):
    """512^3, CIC: the particles of an octant (22 times the time of as many all over the
    box), 1000 in a corner (17 times)."""
    n = 1 << 22
    assert time_us(MASL, uniform(n, part=0.5), 512, 'CIC') <= 3.0 * time_us(MASL, uniform(n), 512, 'CIC')
    assert time_us(MASL, uniform(1000, part=0.01), 512, 'CIC') <= 3.0 * time_us(MASL, uniform(1000), 512, 'CIC')


@pytest.mark.parametrize('mas', ['NGP', 'CIC', 'TSC', 'PCS'])
@pytest.mark.parametrize('dims,lo,hi', [(5, 0.4, 0.6), (8, 0.0, 0.1), (9, 0.9, 0.999), (33, 0.3, 0.4), (64, 0.0, 0.01), (70, 0.99, 0.999)])
def test_gaps_equal_atomic_sums(MASL, mas, dims, lo, hi):
    """Columns and segments before, between and after the particles are empty.  Both
    strategies sum float32 products of the same weights: at most 4000 roundings of 2^-24
    of a cell's value each."""
    pos = uniform(4000, seed=dims) * (hi - lo) + lo * BOX
    w = torch.rand(4000, generator=torch.Generator(device='cuda').manual_seed(7), device='cuda') + 0.5
    for weights in (None, w):
        a, b = torch.zeros((dims,) * 3, device='cuda'), torch.zeros((dims,) * 3, device='cuda')
        MASL.MA(pos, a, BOX, mas, weights, strategy='sorted')
        MASL.MA(pos, b, BOX, mas, weights, strategy='atomic')
        x, y = a.cpu().numpy().astype(np.float64), b.cpu().numpy().astype(np.float64)
        assert np.all(np.abs(x - y) <= 2 * 4000 * 2.0 ** -24 * np.maximum(x, y))


@pytest.mark.parametrize('weighted,bound', [(False, 4.0), (True, 12.0)])
def test_ngp_of_crowded_cells_costs_little(MASL, weighted, bound):
    """16.8 million particles in 343 cells of 128^3 (33 times the time of as many all over
    the box; with masses 28)."""
    n = 1 << 24
    w = torch.ones(n, device='cuda') if weighted else None
    assert time_us(MASL, uniform(n, part=0.05), 128, 'NGP', w) <= bound * time_us(MASL, uniform(n), 128, 'NGP', w)


@pytest.mark.parametrize('base', [0.0, 3.0, -7.0, 0.25, 2.0 ** 24 - 40, 2.0 ** 25])
@pytest.mark.parametrize('counts', [(1, 2, 3, 4, 5), (6, 40, 100, 33, 1)])
def test_ngp_cells_equal_the_serial_sums(MASL, base, counts):
    """Cells of a few to many particles, next to each other along z (a segment's end
    between them), on grid values that are whole or not, below and past 2^24: the bits of
    float32 additions in order."""
    dims = 16
    cells = [(0, 0, 6), (0, 0, 7), (0, 0, 8), (0, 0, 9), (0, 3, 15)]
    pos = np.concatenate([np.tile(np.array(c), (k, 1)) for c, k in zip(cells, counts)]).astype(np.float32)
    rng = np.random.default_rng(3)
    pos = rng.permutation(pos) * np.float32(BOX / dims)
    w = rng.random(len(pos)).astype(np.float32)
    for weights in (None, w):
        ref = np.full((dims,) * 3, base, dtype=np.float32)
        idx = np.rint(pos * (dims / BOX)).astype(int) % dims
        for i, k in enumerate(idx):
            ref[tuple(k)] += np.float32(1.0) if weights is None else weights[i]
        grid = torch.full((dims,) * 3, base, device='cuda')
        MASL.MA(torch.from_numpy(pos).cuda(), grid, BOX, 'NGP', None if weights is None else torch.from_numpy(w).cuda(),
                strategy='sorted')
        assert np.array_equal(grid.cpu().numpy(), ref)


def longest_chain(n, s):
    """Additions that one value passes through at most: 8192 particles of a cell (or their
    255 companions' share of more) in 32 lanes, the lanes and warps, the particles of s
    cells that are walked, the s^2 columns, the grid's value."""
    return 256 + n // 256 + 13 + s * 127 + s * s + 1


@pytest.mark.parametrize('mas', ['CIC', 'TSC', 'PCS'])
@pytest.mark.parametrize('dims,counts', [(1, (300,)), (2, (64, 127, 128, 8192)), (7, (8, 9, 63, 64, 65, 126, 127, 128, 129, 191, 200)),
                                         (33, (8199, 8200, 8201, 8263, 20000, 1, 500)), (64, tuple(range(60, 140)))])
def test_crowded_cells_equal_float64(MASL, mas, dims, counts):
    """Cells of given numbers of particles (around the ends of blocks and the split
    between a warp and a CTA), the first and the last of the box among them, against
    float64 sums of the same float32 positions; the same bits on every run."""
    rng = np.random.default_rng(dims)
    s = {'CIC': 2, 'TSC': 3, 'PCS': 4}[mas]
    cells = rng.choice(dims ** 3, min(len(counts), dims ** 3), replace=False)
    cells[0] = 0
    cells[-1] = dims ** 3 - 1
    base = np.concatenate([np.full(k, c) for c, k in zip(cells, counts)])
    pos = np.stack([base // dims ** 2, base // dims % dims, base % dims], 1) + 0.05 + 0.9 * rng.random((len(base), 3))
    pos = rng.permutation((pos * (BOX / dims)).astype(np.float32))
    w = (rng.random(len(pos)) + 0.5).astype(np.float32)
    for weights in (None, w):
        grids = []
        for _ in range(2):
            a, b = (torch.full((dims,) * 3, 0.5, device='cuda') for _ in range(2))
            MASL.MA(torch.from_numpy(pos).cuda(), a, BOX, mas, None if weights is None else torch.from_numpy(weights).cuda(),
                    interlaced=b, strategy='sorted')
            grids.append((a.cpu().numpy(), b.cpu().numpy()))
        assert np.array_equal(grids[0], grids[1])
        for k, shift in ((0, 0.0), (1, 0.5)):
            x = pos.astype(np.float64) * (dims / BOX) + shift
            ref = np.full(dims ** 3, 0.5)
            first, c = [], []
            for a in range(3):
                if mas == 'CIC':
                    f = np.floor(x[:, a])
                    u = x[:, a] - f
                    first.append(f), c.append([1 - u, u])
                elif mas == 'TSC':
                    f = np.floor(x[:, a] - 0.5)
                    u = x[:, a] - f - 1
                    first.append(f), c.append([0.5 * (0.5 - u) ** 2, 0.75 - u * u, 0.5 * (0.5 + u) ** 2])
                else:
                    f = np.floor(x[:, a]) - 1
                    d = [np.abs(x[:, a] - f - j) for j in range(4)]
                    first.append(f), c.append([np.where(t < 1, (4 - 6 * t * t + 3 * t ** 3) / 6, np.maximum(2 - t, 0) ** 3 / 6) for t in d])
            for l in range(s):
                for m in range(s):
                    for q in range(s):
                        i = [(first[a] + o).astype(int) % dims for a, o in enumerate((l, m, q))]
                        v = c[0][l] * c[1][m] * c[2][q]
                        np.add.at(ref, (i[0] * dims + i[1]) * dims + i[2], v if weights is None else v * weights)
            # a float32 position is off by 2^-24 of the box, dims * 2^-24 cells, and as much
            # again in the product and the shift; a weight's slope is at most 1.  The grid's
            # sum of all particles bounds what that moves in a cell of them.
            slope = 8.0 * dims * 2.0 ** -24 * 1.5 * s
            got = grids[0][k].reshape(-1).astype(np.float64)
            near = np.zeros(dims ** 3)
            for l in range(s):
                for m in range(s):
                    for q in range(s):
                        i = [(first[a] + o).astype(int) % dims for a, o in enumerate((l, m, q))]
                        np.add.at(near, (i[0] * dims + i[1]) * dims + i[2], 1.0)
            tol = (longest_chain(max(counts), s) + 8) * 2.0 ** -24 * ref + slope * near
            assert np.all(np.abs(got - ref) <= tol)


@pytest.mark.parametrize('mas,dims', [('CIC', 128), ('CIC', 256), ('CIC', 512), ('TSC', 256), ('PCS', 256)])
def test_crowded_cells_cost_little(MASL, mas, dims):
    """16.8 million particles in a corner of a twentieth of the box's side (walked one by
    one: 6 to 141 times the time of as many all over the box)."""
    n = 1 << 24
    assert time_us(MASL, uniform(n, part=0.05), dims, mas) <= 4.0 * time_us(MASL, uniform(n), dims, mas)


def test_small_grids_keep_short_walks(MASL):
    """2^20 particles on 32^3 (32 a cell) in little more than the time of 64^3 (1.45 times
    with eight layers a CTA)."""
    pos = uniform(1 << 20)
    assert time_us(MASL, pos, 32, 'CIC') <= 1.2 * time_us(MASL, pos, 64, 'CIC')
